"""The calls by which this engine's speed is followed: powder FIDs through the public entry points.

A case is one spin system class, powder set and acquisition; the couplings, shifts and tensor
orientations come from the seed.  `run` is the call a program makes (`oneFID.FID`,
`oneFID.p2pFID`, or a batch of requests through `Server`), host arrays in and the FID out.
`exact` forms the same FIDs in dense 64-bit torch / numpy from the definition: step
propagators, the period's Dyson products and direct traces, without a Floquet basis.

Keys of a case:
  kind       "mas" (gamma-COMPUTE powder FID), "static", "p2p" (point to point), "serve"
  iso        isotopes of the spins, in order
  powder     crystallites
  steps      steps per rotor period ("mas"); steps per chunk ("p2p")
  points     FID points
  wr         rotor speed, Hz
  mixed      the mixed-precision form (else FP64, the default)
  rho, det   operator expressions
  base, factor, rf   "p2p": chunks per period, chunks per point, windowed 1H decoupling
  jobs       "serve": requests submitted at once
"""
import math
import time

import numpy as np
import torch

import blochlib_gb300 as bl

MAGIC = 54.7356
SPIN = {"1H": 0.5, "13C": 0.5, "15N": 0.5, "2H": 1.0, "23Na": 1.5, "27Al": 2.5}
EXACT_FLOPS = 4e12  # dense 64-bit work up to which exact() is formed (seconds)


# ------------------------------------------------------------------ the cases
def _mas(name, iso, powder, steps, points, wr, mixed, rho="Fx", det="Fp"):
    return dict(name=name, kind="mas", iso=iso, powder=powder, steps=steps, points=points, wr=wr, mixed=mixed,
                rho=rho, det=det)


def _protons(n):
    return " ".join(["1H"] * n)


def listed():
    return [
        # a single crystal, or one orientation inside a caller's own loop: latency alone
        _mas("single_crystal", _protons(3), 1, 64, 1024, 10e3, False),
        # 13C-1H pair on the 1154-point set (the small benchmark configuration)
        _mas("pair", "13C 1H", 1154, 100, 1024, 10e3, False, rho="Ix 0", det="Ip 0"),
        # static pattern of a heteronuclear three-spin group
        dict(name="static", kind="static", iso="13C 1H 1H", powder=1154, steps=1, points=2048, wr=0.0, mixed=False,
             rho="Fx", det="Fp"),
        # point-to-point FID at a rational sampling under windowed 1H decoupling
        dict(name="p2p_rf", kind="p2p", iso="13C 1H 1H", powder=677, steps=4, points=512, wr=12e3, mixed=False,
             rho="Ix 0", det="Ip 0", base=9, factor=7, rf=True),
        # four protons, 3722 crystallites: the plain FP64 benchmark configuration, and its mixed form
        _mas("protons4", _protons(4), 3722, 128, 2048, 20e3, False),
        _mas("protons4_mixed", _protons(4), 3722, 128, 2048, 20e3, True),
        # five protons, initial state on one spin (rho and det not related), odd step count
        _mas("protons5_one_site", _protons(5), 320, 157, 1024, 17e3, False, rho="Ix 0"),
        # six and seven protons: the middle of the batch form's range
        _mas("protons6_mixed", _protons(6), 677, 231, 1024, 23e3, True),
        _mas("protons7", _protons(7), 144, 120, 1024, 30e3, False),
        # eight protons: the headline configuration
        _mas("protons8_mixed", _protons(8), 1154, 200, 4096, 30e3, True),
        # nine protons on a small set: the serving stream's large request
        _mas("protons9_mixed", _protons(9), 32, 120, 1024, 27e3, True),
        # a burst of unequal requests through the serving loop
        dict(name="serve", kind="serve", iso="", powder=0, steps=0, points=1024, wr=0.0, mixed=True, rho="Fx",
             det="Fp", jobs=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["mas"] * 7 + ["static", "p2p", "p2p"])
        mixed = kind != "static" and rng.random() < 0.5
        if kind == "mas":
            iso = rng.choice([_protons(k) for k in range(2, 10)] + [_protons(k) for k in (3, 4, 5, 6, 7)] +
                             ["13C 1H", "13C 1H 1H", "15N 13C 1H 1H", "2H 1H 1H", "23Na 1H", "2H 1H 1H 1H 1H"])
        elif kind == "static":
            iso = rng.choice([_protons(2), _protons(3), _protons(4), "13C 1H", "13C 1H 1H", "2H 1H 1H"])
        else:
            iso = rng.choice([_protons(3), _protons(4), _protons(5), "13C 1H 1H", "13C 1H 1H 1H", "2H 1H"])
        n_spin = len(iso.split())
        c = dict(kind=kind, iso=iso, powder=_log_int(rng, 1, 4096), points=_log_int(rng, 100, 4096),
                 wr=0.0 if kind == "static" else float(round(rng.uniform(5e3, 35e3))), mixed=mixed,
                 rho=rng.choice(["Fx", "Ix 0"]), det="Fp", steps=_log_int(rng, 12, 256))
        if kind == "static":
            c["steps"] = 1
        if kind == "p2p":
            c["steps"] = rng.randint(1, 6)
            c["base"], c["factor"] = rng.choice([(9, 7), (2, 3), (5, 3), (8, 1), (16, 5), (12, 1), (7, 11), (1, 1)])
            c["rf"] = "13C" in iso and rng.random() < 0.6
            c["points"] = min(c["points"], 1024)
        if _cost(c) <= most and _bytes_on_device(c) < 40e9 and n_spin <= 9:
            return c


# ------------------------------------------------------------------ spin systems
def _jobs(case):
    """The single FIDs of a case (a serving burst's requests; else the case itself)."""
    if case["kind"] != "serve":
        return [case]
    out = []
    for k in range(case["jobs"]):
        out.append(dict(kind="mas", iso=_protons((2, 5, 3, 6, 4, 7, 3, 5)[k % 8]),
                        powder=(144, 320, 677, 1154)[(3 * k + k // 4) % 4], steps=(64, 101, 128, 177, 231, 90, 256)[k % 7],
                        points=case["points"], wr=5e3 + 2e3 * ((7 * k) % 16), mixed=case["mixed"], rho=case["rho"],
                        det=case["det"]))
    return out


def _parameters(case, seed):
    """The interactions of a seeded system: dicts of kind C, D, J or Q."""
    rng = np.random.default_rng([int(seed), 0xB10C])
    iso = case["iso"].split()

    def euler():
        return float(rng.uniform(0, 360)), math.degrees(math.acos(rng.uniform(-1, 1))), float(rng.uniform(0, 360))

    terms = []
    for k, name in enumerate(iso):
        ppm = 400.0 if name == "1H" else 100.0
        shift = 0.0 if name == "1H" else float(rng.uniform(-50, 50)) * ppm
        terms.append(dict(t="C", iso=shift, a=float(rng.uniform(0, 10) if name == "1H" else rng.uniform(20, 150)) * ppm,
                          eta=float(rng.uniform(0, 1)), i=k, e=euler()))
    side = 5.0 * max(1.0, (len(iso) / 8.0) ** (1 / 3))  # a cube holding them 1.5 A apart
    xyz = []
    while len(xyz) < len(iso):
        p = rng.uniform(0, side, 3)
        if all(np.linalg.norm(p - q) >= 1.5 for q in xyz):
            xyz.append(p)
    gamma = {"1H": 1.0, "13C": 0.25145, "15N": -0.10136, "2H": 0.15351, "23Na": 0.26452, "27Al": 0.26057}
    for i in range(len(iso)):
        for j in range(i + 1, len(iso)):
            d = xyz[j] - xyz[i]
            r = float(np.linalg.norm(d))
            terms.append(dict(t="D", a=-120.07e3 / r ** 3 * gamma[iso[i]] * gamma[iso[j]], i=i, j=j,
                              e=(math.degrees(math.atan2(d[1], d[0])), math.degrees(math.acos(d[2] / r)), 0.0)))
    for i in range(len(iso)):
        for j in range(i + 1, len(iso)):
            terms.append(dict(t="J", iso=float(rng.uniform(0, 200)), i=i, j=j))
    for k, name in enumerate(iso):
        if SPIN[name] > 0.5:
            terms.append(dict(t="Q", a=float(rng.uniform(20e3, 80e3)), eta=float(rng.uniform(0, 1)), i=k, e=euler()))
    return terms


def _lines(case, terms):
    iso = case["iso"].split()
    out = ["numspin %d" % len(iso)] + ["T %s %d" % (s, k) for k, s in enumerate(iso)]
    for t in terms:
        if t["t"] == "C":
            out.append("C %r %r %r %d %r %r %r" % ((t["iso"], t["a"], t["eta"], t["i"]) + t["e"]))
        elif t["t"] == "D":
            out.append("D %r %d %d %r %r %r" % ((t["a"], t["i"], t["j"]) + t["e"]))
        elif t["t"] == "J":
            out.append("J %r %d %d" % (t["iso"], t["i"], t["j"]))
        else:
            out.append("Q %r %r %d %r %r %r" % ((t["a"], t["eta"], t["i"]) + t["e"]))
    return out


def _powder(count, seed):
    """(phi, theta, gamma, weight): a rank-1 lattice of orientations, rotated by the seed."""
    rng = np.random.default_rng([int(seed), 0x9DE2])
    j = np.arange(count, dtype=np.float64)
    frac = lambda x: x - np.floor(x)  # noqa: E731
    u = rng.uniform(0, 1, 3)
    phi = 2 * np.pi * frac(j * 0.6180339887498949 + u[0])
    theta = np.arccos(2 * frac((j + u[1]) / count) - 1)
    gamma = 2 * np.pi * frac(j * 0.7548776662466927 + u[2])
    return phi, theta, gamma, np.full(count, 1.0 / count)


def _rf(case):
    """Windowed decoupling: 1H rf on in the first five chunks of nine (alternating phase)."""
    on = (5 * case["base"] + 8) // 9
    return [(k, "1H", 50e3, 180.0 * (k % 2), 0.0) for k in range(on)] if case.get("rf") else []


def _sweep(case):
    return case["steps"] * case["wr"] if case["kind"] == "mas" else 100e3


# ------------------------------------------------------------------ the calls
def _prepare_one(case, seed):
    system = bl.SolidSys(_lines(case, _parameters(case, seed)))
    phi, theta, gamma, weight = _powder(case["powder"], seed)
    pw = bl.powder.from_arrays(theta=theta, phi=phi, gamma=gamma, weight=weight)
    return dict(case=case, system=system, pw=pw, ro=system.op(case["rho"]), det=system.op(case["det"]))


def prepare(case, seed):
    jobs = [_prepare_one(c, int(seed) + 1000 * k) for k, c in enumerate(_jobs(case))]
    # the serving program keeps its server; the others keep the system, powder and operators
    return dict(case=case, jobs=jobs, server=bl.Server() if case["kind"] == "serve" else None)


def _stored(case, fid):
    """The mixed form's FID (stated to 1e-6 of FP64) as processing programs store it."""
    return fid.astype(np.complex64) if case["mixed"] else fid


def run(state):
    if state["server"] is not None:
        return _run_serve(state)
    s = state["jobs"][0]
    c = s["case"]
    if c["kind"] == "p2p":
        drv = bl.oneFID(s["system"], c["points"], wr=c["wr"], rotb=MAGIC, precision=int(c["mixed"]))
        chunk = 1.0 / (c["wr"] * c["base"])
        fid = drv.p2pFID(s["pw"], s["ro"], s["det"], c["base"], c["factor"], maxtstep=chunk / (c["steps"] - 0.5),
                         rf_chunks=_rf(c))
    else:
        drv = bl.oneFID(s["system"], c["points"], _sweep(c), c["wr"], MAGIC, precision=int(c["mixed"]))
        fid = drv.FID(s["pw"], s["ro"], s["det"])
    return _stored(c, fid)


def _run_serve(state):
    srv = state["server"]
    tickets = []
    for s in state["jobs"]:
        c = s["case"]
        tickets.append(srv.submit(s["system"], s["pw"], s["ro"], s["det"], c["points"], _sweep(c), c["wr"], MAGIC,
                                  precision=int(c["mixed"])))
    out = []
    for s, t in zip(state["jobs"], tickets):
        while True:
            st, fid, _, _ = srv.result(t)
            if st >= bl.Server.DONE:
                break
            time.sleep(1e-4)
        out.append(_stored(s["case"], fid))
    return out


# ------------------------------------------------------------------ work
def _sectors(case):
    """Index lists of equal total Fz (one list under an rf schedule, which mixes them)."""
    dims = [int(2 * SPIN[s] + 1) for s in case["iso"].split()]
    m = np.zeros(1)
    for d in dims:
        m = (m[:, None] + ((d - 1) / 2 - np.arange(d))[None, :]).reshape(-1)
    if case.get("rf"):
        return [np.arange(len(m))]
    return [np.nonzero(m == v)[0] for v in sorted(set(m.tolist()), reverse=True)]


def _counts(case):
    b = [len(s) for s in _sectors(case)]
    s3 = sum(x ** 3 for x in b)
    pairs = list(zip(b, b[1:])) if len(b) > 1 else [(b[0], b[0])]
    return sum(b), s3, sum(x * x for x in b), sum(x * y * (x + y) for x, y in pairs), sum(x * y for x, y in pairs)


def _flops(case):
    """A matrix exponential (11 b^3) and one product per step, the period's eigenvectors, the
    transforms of det, one correlation per element (two transforms) and the FID's sums."""
    n_dim, s3, _, q3, q2 = _counts(case)
    n = case["steps"] * case.get("base", 1)
    if case["kind"] == "static":
        return case["powder"] * (11.0 * s3 + 16.0 * q3 + 8.0 * case["points"] * q2)
    per = n * (11.0 * s3 + 8.0 * s3 + 8.0 * s3 + 8.0 * q3) + 100.0 * s3 + 8.0 * case["points"] * q2
    if case["kind"] == "mas":
        per += q2 * 2 * 5.0 * 2 * n * math.log2(max(2, 2 * n))
    return case["powder"] * per


def _cost(case):
    """Seconds, roughly (FP64 at 1 TFLOP/s; the mixed form 3 to 9 times that, by block size)."""
    if case["kind"] == "serve":
        return sum(_cost(c) for c in _jobs(case))
    b = max(len(s) for s in _sectors(case))
    return _flops(case) / 1e12 / ((3.0 if b > 74 else 9.0 if b >= 20 else 4.0) if case["mixed"] else 1.0)


def _bytes_on_device(case):
    n = case["steps"] * case.get("base", 1)
    _, _, s2, _, q2 = _counts(case)
    return 16.0 * case["powder"] * (n * (2.5 * s2 + 2 * q2) + case["points"] / max(n, 1) * q2)


def work(case):
    total = dict(bytes=0.0, flops=0.0)
    for c in _jobs(case):
        n_dim = sum(len(s) for s in _sectors(c))
        total["bytes"] += 32.0 * c["powder"] + 32.0 * n_dim * n_dim + (8.0 if c["mixed"] else 16.0) * c["points"]
        total["flops"] += _flops(c)
    return total


# ------------------------------------------------------------------ 64-bit reference
def _operators(case):
    """{name: [dense operator of each spin]} in the product basis, spin 0 slowest."""
    dims = [int(2 * SPIN[s] + 1) for s in case["iso"].split()]
    ops = {"x": [], "y": [], "z": [], "p": []}
    for k, d in enumerate(dims):
        m = (d - 1) / 2 - np.arange(d)
        p = np.zeros((d, d))
        s = (d - 1) / 2
        for r in range(d - 1):
            p[r, r + 1] = math.sqrt(s * (s + 1) - m[r + 1] * (m[r + 1] + 1))
        one = {"z": np.diag(m), "p": p, "x": (p + p.T) / 2, "y": (p - p.T) / 2j}
        for name, o in one.items():
            left, right = int(np.prod(dims[:k])), int(np.prod(dims[k + 1:]))
            ops[name].append(np.kron(np.kron(np.eye(left), o), np.eye(right)))
    return ops


def _expression(ops, expr):
    name, _, spin = expr.partition(" ")
    which = name[1]
    return ops[which][int(spin)] if name[0] == "I" else sum(ops[which])


def _euler(a, b, g):
    ca, sa, cb, sb, cg, sg = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(g), np.sin(g)
    z = np.zeros_like(cb * ca * cg)
    return np.array([[ca * cb * cg - sa * sg, sa * cb * cg + ca * sg, -sb * cg + z],
                     [-ca * cb * sg - sa * cg, -sa * cb * sg + ca * cg, sb * sg + z],
                     [ca * sb + z, sa * sb + z, cb + z]])


def _hamiltonian_terms(case, terms, ops):
    """(constant part, tensors (K, 3, 3), operators (K, N, N)) of H = Hc + sum_k (v P_k v) T_k."""
    iso = case["iso"].split()
    n = len(ops["z"][0])
    hc, pas, top = np.zeros((n, n)), [], []
    for t in terms:
        z = ops["z"]
        if t["t"] == "J":
            hc = hc + t["iso"] * z[t["i"]] @ z[t["j"]]
            continue
        rot = _euler(*np.radians(t["e"]))
        if t["t"] == "C":
            hc = hc - t["iso"] * z[t["i"]]
            diag, op = np.array([(t["eta"] - 1) / 2, -(t["eta"] + 1) / 2, 1.0]) * t["a"], z[t["i"]]
        elif t["t"] == "D":
            zz = z[t["i"]] @ z[t["j"]]
            if iso[t["i"]] == iso[t["j"]]:
                xx, yy = ops["x"][t["i"]] @ ops["x"][t["j"]], (ops["y"][t["i"]] @ ops["y"][t["j"]]).real
                op = 2 * zz - xx - yy
            else:
                op = 2 * zz
            diag = np.array([-0.5, -0.5, 1.0]) * t["a"]
        else:
            s = SPIN[iso[t["i"]]]
            diag = np.array([(t["eta"] - 1) / 2, -(t["eta"] + 1) / 2, 1.0]) * t["a"] / (4 * s * (2 * s - 1))
            op = 3 * z[t["i"]] @ z[t["i"]]
        pas.append(rot @ np.diag(diag) @ rot.T)
        top.append(op)
    return hc, np.array(pas), np.array(top)


def _rotor_row(rows, phases):
    """Third rows (C, n, 3) of R_rotor(phase) R_powder."""
    tilt = math.radians(MAGIC)
    rp = _euler(rows[0], rows[1], rows[2]).transpose(2, 0, 1)
    rr = np.stack([np.sin(phases) * math.sin(tilt), -np.cos(phases) * math.sin(tilt),
                   np.full_like(phases, math.cos(tilt))], axis=1)
    return np.einsum("ia,cab->cib", rr, rp)


def _exact_one(case, seed):
    n_dim, s3, s2, q3, q2 = _counts(case)
    n = case["steps"] * case.get("base", 1)
    periods = case["points"] / n if case["kind"] == "mas" else 1.0
    dense = case["powder"] * 8.0 * (n * 14.0 * s3 + (n * (periods + 2.0) * 2.0 + (2.0 * case["points"] if case["kind"] == "p2p" else 0.0)) * q3)
    if dense + 100.0 * case["powder"] * n * periods * q2 > EXACT_FLOPS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    terms, ops = _parameters(case, seed), _operators(case)
    hc, pas, top = _hamiltonian_terms(case, terms, ops)
    rows, sectors = _powder(case["powder"], seed), _sectors(case)
    rho, det = _expression(ops, case["rho"]).astype(complex), _expression(ops, case["det"]).astype(complex)
    if case["kind"] == "static":
        return _exact_static(case, hc, pas, top, rows, sectors, rho, det)
    tau = 1.0 / case["wr"] / n
    phases = (np.arange(n) + 0.5) * tau * case["wr"] * 2 * np.pi
    row = _rotor_row(rows, phases)
    coef = np.einsum("cia,kab,cib->cik", row, pas, row, optimize=True)
    extra = np.zeros((case.get("base", 1),) + hc.shape, complex)  # the rf of each chunk
    for chunk, name, amp, ph, off in _rf(case) if case["kind"] == "p2p" else []:
        for k, s in enumerate(case["iso"].split()):
            if s == name:
                extra[chunk] += amp * (ops["x"][k] * math.cos(math.radians(ph)) + ops["y"][k] * math.sin(math.radians(ph)))
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731
    rosym = np.array_equal(rho, 0.5 * (det + det.conj().T))
    fid = torch.zeros(case["points"], dtype=torch.complex128, device=dev)
    length = (-(-case["points"] // n) + 1) * n if case["kind"] == "mas" else n
    per_c = 16.0 * (n * s2 * 8 + length * q2 * 6)
    step = max(1, min(case["powder"], int((8e9 if dev == "cuda" else 1e9) / per_c)))
    for c0 in range(0, case["powder"], step):
        w = t(rows[3][c0:c0 + step])
        prods = []  # per sector: A_1 .. A_n (C, n, b, b)
        for sec in sectors:
            ix = np.ix_(sec, sec)
            h = torch.einsum("cik,kxy->cixy", t(coef[c0:c0 + step]), t(top[:, ix[0], ix[1]])).to(torch.complex128)
            h = h + t(np.repeat(hc[ix] + extra[:, ix[0], ix[1]], case["steps"] if case["kind"] == "p2p" else n, axis=0))
            u = torch.linalg.matrix_exp(-2j * math.pi * tau * h)
            a = [u[:, 0]]
            for i in range(1, n):
                a.append(u[:, i] @ a[-1])
            prods.append(torch.stack(a, 1))
        part = (_exact_mas if case["kind"] == "mas" else _exact_p2p)(case, prods, sectors, t, rho, det, rosym, w, n)
        fid += part
    return fid.cpu().numpy()


def _blocks(m, sectors):
    """Pairs (a, b, block) of sectors where the operator is not zero."""
    return [(a, b, m[np.ix_(x, y)]) for a, x in enumerate(sectors) for b, y in enumerate(sectors)
            if np.any(m[np.ix_(x, y)])]


def _exact_mas(case, prods, sectors, t, rho, det, rosym, w, n):
    """fid[k] = s sum_i Tr(X[k + i] R_i): X[jn + m] = F^j Q_m F^-j, Q_m and R_m the transforms of
    det and rho (Q + Q^H when rho = (det + det^H)/2) by A_(m+1), F = A_n; one long correlation."""
    points = case["points"]
    periods = -(-points // n) + 1
    size = 1 << (periods * n + n - 1).bit_length()
    left = {(a, b): prods[a].mH @ t(m) @ prods[b] for a, b, m in _blocks(det, sectors)}
    if rosym:
        right = {}
        for (a, b), q in left.items():
            for key, v in (((a, b), q), ((b, a), q.mH)):
                right[key] = right[key] + v if key in right else v
    else:
        right = {(a, b): prods[a].mH @ t(m) @ prods[b] for a, b, m in _blocks(rho, sectors)}
    total = torch.zeros(size, dtype=torch.complex128, device=w.device)
    for (a, b), q in left.items():
        if (b, a) not in right:
            continue
        fa, fb = prods[a][:, -1:], prods[b][:, -1:].mH
        x = [q]
        for _ in range(periods - 1):
            x.append(fa @ x[-1] @ fb)
        x = torch.cat(x, 1).flatten(2).transpose(1, 2).contiguous()          # (C, elements, time)
        r = right[(b, a)].transpose(2, 3).flatten(2).transpose(1, 2).contiguous()
        for e in range(0, x.shape[1], 64):
            fx = torch.fft.fft(x[:, e:e + 64], size)
            fr = torch.fft.fft(r[:, e:e + 64].conj(), size).conj()
            total += torch.einsum("cef,cef,c->f", fx, fr, w.to(torch.complex128))
    return torch.fft.ifft(total)[:points] / (n // (2 if rosym else 1))


def _exact_p2p(case, prods, sectors, t, rho, det, rosym, w, n):
    """fid[p] = Tr(det G rho G^H) / Tr(det det^H), G the propagator over p * factor chunks."""
    base, factor, sub = case["base"], case["factor"], case["steps"]
    heis = {}
    dets = _blocks(det, sectors)
    for j in range(1, base + 1):
        heis[j] = [(a, b, prods[a][:, j * sub - 1].mH @ t(m) @ prods[b][:, j * sub - 1]) for a, b, m in dets]
    cur = {(a, b): t(m).expand(len(w), *m.shape) for a, b, m in _blocks(rho, sectors)}
    out, q_now = [], 0
    for p in range(case["points"]):
        m = p * factor
        if m == 0:
            q, ops = 0, [(a, b, t(x).expand(len(w), *x.shape)) for a, b, x in dets]
        else:
            j = (m - 1) % base + 1
            q, ops = (m - j) // base, heis[j]
        while q_now < q:
            cur = {(a, b): prods[a][:, -1] @ x @ prods[b][:, -1].mH for (a, b), x in cur.items()}
            q_now += 1
        v = sum((x * cur[(b, a)].transpose(1, 2)).sum((1, 2)) for a, b, x in ops if (b, a) in cur)
        out.append((v * w).sum() if not isinstance(v, int) else w.sum() * 0j)
    return torch.stack(out) / float(np.sum(np.abs(det) ** 2))


def _exact_static(case, hc, pas, top, rows, sectors, rho, det):
    """fid[k] = sum_rs A_rs B_rs^k in the eigenbasis; terms with |A|^2 <= 1e-10 are left out."""
    row = _rotor_row(rows, np.zeros(1))
    coef = np.einsum("cia,kab,cib->ck", row, pas, row, optimize=True)
    vec, val = [], []
    for sec in sectors:
        ix = np.ix_(sec, sec)
        h = hc[ix] + np.einsum("ck,kxy->cxy", coef, top[:, ix[0], ix[1]])
        e, v = np.linalg.eigh(h)
        vec.append(v), val.append(e)
    fid = np.zeros(case["points"], complex)
    right = {(a, b): m for a, b, m in _blocks(rho, sectors)}
    k = np.arange(case["points"])
    for a, b, m in _blocks(det, sectors):
        if (b, a) not in right:
            continue
        d = vec[a].transpose(0, 2, 1) @ m @ vec[b]
        s = vec[b].transpose(0, 2, 1) @ right[(b, a)] @ vec[a]
        amp = d * s.transpose(0, 2, 1)
        amp = np.where(np.abs(amp) ** 2 <= 1e-10, 0, amp) * rows[3][:, None, None]
        freq = (val[a][:, :, None] - val[b][:, None, :]) * 2 * np.pi / _sweep(case)
        amp, freq = amp.reshape(-1), freq.reshape(-1)
        for c0 in range(0, len(amp), 4096):
            fid += amp[c0:c0 + 4096] @ np.exp(1j * freq[c0:c0 + 4096, None] * k[None, :])
    return fid


def exact(case, seed):
    got = [_exact_one(c, int(seed) + 1000 * k) for k, c in enumerate(_jobs(case))]
    return got if case["kind"] == "serve" else got[0]
