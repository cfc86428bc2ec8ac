"""Workloads of the contraction library, from one small correlator to the largest
lattices of its benchmark, each run through the public entry points.

A case names an operation (``op``), a lattice (``lx, ly, lz, lt``; PyQUDA even/odd
site order), a storage type (``dtype``: "c128", the drop-in format, or "c64", the
mixed form) and the operation's options.  Propagators are a part common to every
site plus site noise, times exp(-m |t - t0|): correlators then carry a signal on
top of noise, as real ones do.

Correlators of the mixed form come back in complex128 buffers but carry the
accuracy of FP32 arithmetic; a program that works in complex64 keeps them in
complex64, and so does ``run``.
"""
import ctypes

import numpy as np
import torch

from contract_gb300 import _lib, api, pycontract as pc

DEVICE = "cuda:0"
MASS = {"u": 0.20, "d": 0.25, "s": 0.30}


# ------------------------------------------------------------------- the cases --

def listed():
    return [
        # One correlator of a test lattice through the drop-in call: what counts is the call and its launch.
        dict(name="meson_small", op="meson", dtype="c128", lx=4, ly=4, lz=4, lt=8, gamma_a=15, gamma_b=15),
        # A meson spectrum: 16 sink structures for one source, per site, the drop-in call on a production-like volume.
        dict(name="meson_all_c128", op="meson_all", dtype="c128", lx=16, ly=16, lz=16, lt=32, gamma_a=5, source=True,
             summed=False),
        # The same spectrum in the mixed form, summed per timeslice, on a lattice whose extents divide by nothing much.
        dict(name="meson_all_c64_odd", op="meson_all", dtype="c64", lx=18, ly=13, lz=22, lt=45, gamma_a=15,
             source=False, summed=True),
        # The reference's baryon example: six contraction types, one call each, positive-parity projector, per site.
        dict(name="baryon_dropin_c128", op="baryon_types", dtype="c128", lx=24, ly=24, lz=24, lt=32, gamma_a=5,
             gamma_b=5, proj="parity"),
        # One contraction type with a gamma matrix in the open slot, mixed form, per timeslice, odd extents.
        dict(name="baryon_one_c64_odd", op="baryon", dtype="c64", lx=22, ly=17, lz=25, lt=54, gamma_a=5, gamma_b=5,
             type=3, proj="gamma", summed=True),
        # A whole baryon correlator (six types, both parities) on a small lattice: a call of a few launches.
        dict(name="baryon_all_small", op="baryon_all", dtype="c64", lx=8, ly=8, lz=8, lt=16, gamma_a=5, gamma_b=5,
             proj="both", same=False),
        # The benchmark: six types, both parities, 24^3 x 64, mixed form.
        dict(name="baryon_all_c64", op="baryon_all", dtype="c64", lx=24, ly=24, lz=24, lt=64, gamma_a=5, gamma_b=5,
             proj="both", same=False),
        # The same pass in double precision.
        dict(name="baryon_all_c128", op="baryon_all", dtype="c128", lx=16, ly=16, lz=16, lt=48, gamma_a=5, gamma_b=5,
             proj="both", same=False),
        # A sequential source for a three-point function: a propagator-sized result in the slot of one quark.
        dict(name="sequential_c64", op="sequential", dtype="c64", lx=32, ly=32, lz=32, lt=48, gamma_a=5, gamma_b=5,
             gamma_c=8, type=1, slot=2),
        # All 256 meson pairs at 125 momenta, mixed form: the largest projection of the benchmark.
        dict(name="momentum_c64", op="momentum", dtype="c64", lx=32, ly=32, lz=32, lt=64, nmax=2, same=False),
        # The projection in double precision on uneven extents.
        dict(name="momentum_c128_odd", op="momentum", dtype="c128", lx=18, ly=15, lz=20, lt=28, nmax=2, same=False),
        # Many sources at once on three lattices (nucleon and pion share the u quark): one batched call.
        dict(name="batch_c64", op="batch", dtype="c64", lx=16, ly=16, lz=16, lt=32, nmax=1, same=True, sources=7),
    ]


def draw(rng):
    """One more case of the listed ranges: any operation, both storage types, odd extents among even ones."""
    op = rng.choice(["meson", "meson_all", "baryon", "baryon_types", "baryon_all", "baryon_all", "sequential",
                     "diquark", "momentum", "momentum", "batch"])
    c128 = op != "batch" and rng.random() < 0.4 or op == "baryon_types"
    most = {"meson": 600_000, "meson_all": 300_000, "baryon": 300_000, "baryon_types": 200_000, "baryon_all": 200_000,
            "sequential": 200_000, "diquark": 200_000, "momentum": 150_000}.get(op) if c128 else \
        {"momentum": 1_500_000, "batch": 60_000}.get(op, 1_200_000)
    least = {"momentum": 2_000, "batch": 4_000}.get(op, 512)
    volume = int(least * (most / least) ** rng.random())
    lt = max(4, min(64, int(round(2 * volume ** 0.25 * rng.uniform(0.7, 1.4)))))
    low = 5 if op in ("momentum", "batch") else 3
    side = (volume / lt) ** (1 / 3)
    lx = 2 * max((low + 1) // 2, min(16, int(round(side * rng.uniform(0.75, 1.3) / 2))))
    ly = max(low, min(40, int(round(side * rng.uniform(0.75, 1.3)))))
    lz = max(low, min(40, int(round(volume / (lt * lx * ly)))))
    case = dict(op=op, dtype="c128" if c128 else "c64", lx=lx, ly=ly, lz=lz, lt=lt)
    g = [5, 5, 5, 15, 10, 7, 13]
    if op in ("meson", "meson_all"):
        case["gamma_a"] = rng.randrange(16)
        if op == "meson":
            case["gamma_b"] = rng.randrange(16)
        else:
            case["source"] = rng.random() < 0.5
        if op == "meson_all":
            case["summed"] = rng.random() < 0.5
    elif op in ("baryon", "baryon_types", "baryon_all"):
        case["gamma_a"], case["gamma_b"] = rng.choice(g), rng.choice(g)
        case["proj"] = rng.choice(["both", "both", "parity", "polarised", "dense"]) if op == "baryon_all" \
            else rng.choice(["gamma", "parity", "parity", "polarised", "dense"])
        if op == "baryon":
            case["type"] = rng.randrange(6)
            case["summed"] = rng.random() < 0.6
        if op == "baryon_all":
            case["same"] = rng.random() < 0.4
    elif op in ("sequential", "diquark"):
        case["gamma_a"], case["gamma_b"] = rng.choice(g), rng.choice(g)
        if op == "sequential":
            case.update(gamma_c=rng.choice([0, 8, 8, 7]), type=rng.randrange(6), slot=rng.randrange(3))
    elif op == "momentum":
        case.update(nmax=rng.choice([0, 1, 2, 2]), same=rng.random() < 0.4)
    else:
        case.update(nmax=1, same=rng.random() < 0.7, sources=rng.randint(2, 8))
    return case


# ------------------------------------------------------------------ their inputs --

def _latt(case):
    return (case["lx"], case["ly"], case["lz"], case["lt"])


def _volume(latt):
    return latt[0] * latt[1] * latt[2] * latt[3]


def _dtype(case):
    return torch.complex128 if case["dtype"] == "c128" else torch.complex64


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _normal(g, shape, double):
    x = torch.randn(shape, generator=g, device=DEVICE)
    if not double:
        return x
    # a full mantissa: the low bits of a second number
    return x.double() + torch.randn(shape, generator=g, device=DEVICE).double() * 2.0 ** -26


def _propagator(latt, seed, flavour, dtype):
    """[V, 4, 4, 3, 3]: exp(-m |t|) (W + noise(x)) / sqrt 2, W the same at every site."""
    lx, ly, lz, lt = latt
    double = dtype == torch.complex128
    g = _generator(seed * 7919 + ord(flavour))
    p = _normal(g, (_volume(latt), 288), double)
    p += _normal(g, (288,), double)
    t = torch.arange(_volume(latt), device=DEVICE) // (lx * ly * lz // 2) % lt
    far = torch.minimum(t, lt - t)
    p *= (0.5 ** 0.5 * torch.exp(-MASS[flavour] * far.double())).to(p.dtype)[:, None]
    return torch.view_as_complex(p.view(-1, 144, 2)).view(-1, 4, 4, 3, 3)


def _projectors(kind):
    """The projectors W[m][n] of the open spin slot, [n, 4, 4]."""
    e, gm = np.eye(4), _gammas()
    plus, minus = (e + gm[8]) / 2, (e - gm[8]) / 2
    if kind == "both":
        return np.stack([plus, minus])
    if kind == "parity":
        return plus[None]
    if kind == "polarised":
        return (plus @ (e - 1j * gm[1] @ gm[2]) / 2)[None]
    if kind == "dense":
        k = np.arange(16.0).reshape(4, 4)
        return (np.cos(1 + k * 1.7) + 1j * np.sin(0.3 + k * k * 0.61))[None]
    return gm[8][None]


def _momenta(nmax):
    r = range(-nmax, nmax + 1)
    return np.array([(x, y, z) for z in r for y in r for x in r], dtype=np.int32)


class _MesonItem(ctypes.Structure):
    _fields_ = [("propag_i", ctypes.c_void_p), ("propag_j", ctypes.c_void_p), ("correl", ctypes.c_void_p),
                ("lattice", ctypes.c_int * 4)]


class _BaryonItem(ctypes.Structure):
    _fields_ = [("propag_i", ctypes.c_void_p), ("propag_j", ctypes.c_void_p), ("propag_n", ctypes.c_void_p),
                ("correl", ctypes.c_void_p), ("lattice", ctypes.c_int * 4)]


def _ints(values):
    return (ctypes.c_int * len(values))(*[int(v) for v in values])


def _batch_lattices(case):
    """The lattice of each source: the case's, one about 1.5 times as wide, one twice as wide, in the proportion of
    a scan over three ensembles (most sources on the smallest)."""
    lx, ly, lz, lt = _latt(case)
    middle = (2 * (lx * 3 // 4), ly * 3 // 2, lz * 3 // 2, lt * 3 // 2)
    wide = (2 * lx, 2 * ly, 2 * lz, 2 * lt)
    n = case["sources"]
    wides = n // 7
    middles = (n - wides) // 3
    return [_latt(case)] * (n - wides - middles) + [middle] * middles + [wide] * wides


def _sources(case, seed):
    """Per source of a batch: its lattice, the u quarks of slots i and j (one field or two) and the d quark."""
    out = []
    for k, latt in enumerate(_batch_lattices(case)):
        s = seed * 1009 + k
        u = _propagator(latt, s, "u", torch.complex64)
        v = u if case["same"] else _propagator(latt, s + 500_009, "u", torch.complex64)
        out.append((latt, u, v, _propagator(latt, s, "d", torch.complex64)))
    return out


def _props(case, seed):
    """The propagators that the case's operation reads, in the order of its arguments."""
    latt, dt = _latt(case), _dtype(case)
    first = _propagator(latt, seed, "u", dt)
    same = case.get("same", False)
    if case["op"] in ("meson", "meson_all", "momentum", "diquark"):
        return [first, first if same else _propagator(latt, seed, "s", dt)]
    second = first if same else _propagator(latt, seed + 500_009, "u", dt)
    return [first, second, _propagator(latt, seed, "d", dt)]


def prepare(case, seed):
    state = {"case": case, "latt": _latt(case)}
    if case["op"] == "batch":
        moms = _momenta(case["nmax"])
        src = _sources(case, seed)
        state.update(keep=src, moms=moms)
        state["baryon"] = [torch.empty((6, 2, s[0][3]), dtype=torch.complex128, device=DEVICE) for s in src]
        state["meson"] = [torch.empty((len(moms), s[0][3], 256), dtype=torch.complex128, device=DEVICE) for s in src]
        bi, mi = (_BaryonItem * len(src))(), (_MesonItem * len(src))()
        for k, (latt, u, v, d) in enumerate(src):
            bi[k] = _BaryonItem(u.data_ptr(), v.data_ptr(), d.data_ptr(), state["baryon"][k].data_ptr(), _ints(latt))
            mi[k] = _MesonItem(u.data_ptr(), v.data_ptr(), state["meson"][k].data_ptr(), _ints(latt))
        state.update(baryon_items=bi, meson_items=mi,
                     projectors=np.ascontiguousarray(_projectors("both").astype(np.complex128)))
        return state
    state["p"] = _props(case, seed)
    if "proj" in case:
        w = _projectors(case["proj"])
        state["w"] = w.reshape(len(w), 16) if case["op"] == "baryon_all" else w[0]
    if case["op"] == "momentum":
        moms = _momenta(case["nmax"])
        state.update(moms=moms, out=torch.empty((len(moms), case["lt"], 256), dtype=torch.complex128, device=DEVICE))
    return state


# ---------------------------------------------------------------------- one pass --

def _kept(out, case):
    return out if case["dtype"] == "c128" else out.to(torch.complex64)


def _int_p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def run(state):
    c, latt, p = state["case"], state["latt"], state.get("p")
    op = c["op"]
    if op == "meson":
        return _kept(pc.mesonTwoPoint(p[0], p[1], c["gamma_a"], c["gamma_b"]), c)
    if op == "meson_all":
        if c["summed"]:
            return _kept(api.meson_all_timeslice(p[0], p[1], latt, c["gamma_a"], source=c["source"]), c)
        f = pc.mesonAllSourceTwoPoint if c["source"] else pc.mesonAllSinkTwoPoint
        return _kept(f(p[0], p[1], c["gamma_a"]), c)
    if op == "baryon_types":
        return [pc.baryonTwoPoint(*p, t, c["gamma_a"], c["gamma_b"], state["w"]) for t in pc.BaryonContractType]
    if op == "baryon":
        open_slot = dict(gamma_mn=8) if c["proj"] == "gamma" else dict(project_mn=state["w"])
        return _kept(api.baryon(*p, c["type"], c["gamma_a"], c["gamma_b"], latt=latt if c["summed"] else None,
                                **open_slot), c)
    if op == "baryon_all":
        return _kept(api.baryon_all_types(*p, c["gamma_a"], c["gamma_b"], state["w"], latt=latt), c)
    if op == "sequential":
        return pc.baryonSequentialTwoPoint(*p, c["type"], c["slot"], c["gamma_a"], c["gamma_b"], c["gamma_c"])
    if op == "diquark":
        return pc.baryonDiquark(*p, c["gamma_a"], c["gamma_b"])
    lib = _lib.lib()
    if op == "momentum":
        prec = pc.CONTRACT_C128 if c["dtype"] == "c128" else pc.CONTRACT_C64
        lib.contract_meson_all_gamma_momentum(state["out"].data_ptr(), p[0].data_ptr(), p[1].data_ptr(), _volume(latt),
                                              _ints(latt), _int_p(state["moms"]), len(state["moms"]), prec)
        return _kept(state["out"], c)
    lib.contract_batch_mixed(state["baryon_items"], len(state["keep"]), 5, 5, 2, state["projectors"].ctypes.data,
                             state["meson_items"], len(state["keep"]), _int_p(state["moms"]), len(state["moms"]),
                             pc.CONTRACT_C64)
    return {"baryon": [_kept(b, c) for b in state["baryon"]], "meson": [_kept(m, c) for m in state["meson"]]}


# ------------------------------------------------------------- what a pass needs --

def work(case):
    """Bytes: each propagator read once and each result written once.  Flops: complex multiply-adds (8 flops) of the
    products no form of the contraction avoids -- a colour wedge is 36 and a colour dot 9 of them."""
    op, v, lt = case["op"], _volume(_latt(case)), case["lt"]
    item = 16 if case["dtype"] == "c128" else 8
    site = 144 * item
    fields = 1 if case.get("same") else 2
    kept = item  # an output value, as the program keeps it
    if op == "meson":
        return {"bytes": v * (2 * site + kept), "flops": 8.0 * v * 144}
    if op == "meson_all":
        return {"bytes": v * 2 * site + 16 * kept * (lt if case["summed"] else v), "flops": 8.0 * v * 576}
    if op == "baryon":
        return {"bytes": v * 3 * site + kept * (lt if case["summed"] else v), "flops": 8.0 * v * 16 * 45}
    if op == "baryon_types":
        return {"bytes": v * (3 * site + 6 * kept), "flops": 8.0 * v * (64 * 36 + 6 * 16 * 9)}
    if op == "baryon_all":
        n = len(_projectors(case["proj"]))
        wedges = 32 if case["same"] else 64
        return {"bytes": v * (fields + 1) * site + 6 * n * lt * kept, "flops": 8.0 * v * (wedges * 36 + n * 2 * 16 * 9)}
    if op in ("sequential", "diquark"):
        return {"bytes": v * 3 * site, "flops": 8.0 * v * 16 * 36}
    n = (2 * case["nmax"] + 1) ** 3
    if op == "momentum":
        dots = 136 if case["same"] else 256
        return {"bytes": v * fields * site + n * lt * 256 * kept, "flops": 8.0 * v * (dots * 9 + 256)}
    total = {"bytes": 0, "flops": 0.0}
    for latt in _batch_lattices(case):
        w, m = _volume(latt), latt[3]
        total["bytes"] += w * (fields + 1) * site + (12 + 256 * n) * m * kept
        total["flops"] += 8.0 * w * ((32 if case["same"] else 64) * 36 + 2 * 2 * 16 * 9 +
                                     (136 if case["same"] else 256) * 9 + 256)
    return total


# --------------------------------------------------- the same results in 64 bits --

def _gammas():
    """Gamma(n) = g1^(n&1) g2^(n>>1&1) g3^(n>>2&1) g4^(n>>3&1), DeGrand-Rossi basis."""
    i = 1j
    base = [np.array(m, dtype=np.complex128) for m in (
        [[0, 0, 0, i], [0, 0, i, 0], [0, -i, 0, 0], [-i, 0, 0, 0]],
        [[0, 0, 0, -1], [0, 0, 1, 0], [0, 1, 0, 0], [-1, 0, 0, 0]],
        [[0, 0, i, 0], [0, 0, 0, -i], [-i, 0, 0, 0], [0, i, 0, 0]],
        [[0, 0, 1, 0], [0, 0, 0, 1], [1, 0, 0, 0], [0, 1, 0, 0]])]
    out = []
    for n in range(16):
        m = np.eye(4, dtype=np.complex128)
        for bit in range(4):
            if n >> bit & 1:
                m = m @ base[bit]
        out.append(m)
    return np.stack(out)


def _matrix(m):
    return torch.tensor(m, dtype=torch.complex128, device=DEVICE)


EPS = [(0, 1, 2, 1), (1, 2, 0, 1), (2, 0, 1, 1), (0, 2, 1, -1), (2, 1, 0, -1), (1, 0, 2, -1)]
# contraction types: second spin index of P_i, of P_j, and of P_n (first index m), as baryon einsum strings name them
TYPES = ["kln", "knl", "lkn", "lnk", "nkl", "nlk"]
CHUNK = 1 << 17


def _chunks(v):
    return [slice(a, min(v, a + CHUNK)) for a in range(0, v, CHUNK)]


def _wedge(spin, x, y, shape):
    """out[.., s, t, a, d] = sum eps_abc eps_def spin(x[.., b, e], y[.., c, f]), over colours."""
    out = torch.zeros(shape, dtype=torch.complex128, device=DEVICE)
    for a, b, c, s in EPS:
        for d, e, f, r in EPS:
            out[..., a, d] += s * r * spin(x[..., b, e], y[..., c, f])
    return out


def _open_diquark(pi, pj, gij):
    """G[x][s][t][c][f] = sum_ij Gamma_ij[i][j] (P_i[i][s] ^ P_j[j][t]), every baryon type's common part."""
    gi = torch.einsum("ij,xisbe->xjsbe", gij, pi)
    return _wedge(lambda u, w: torch.einsum("xjs,xjt->xst", u, w), gi, pj, (len(pi), 4, 4, 3, 3))


def _baryon_site(g, pn, t, gkl, w):
    """C(x) of one type from G, for P_n with the open slot's matrix W[n][m]."""
    si, sj, sn = TYPES[t]
    n = torch.einsum("nm,xmtcf->xntcf", w, pn)
    if sn == "n":  # P_n closed on itself
        q = torch.einsum("xnncf->xcf", n)
        d = torch.einsum(f"kl,x{si}{sj}cf->xcf", gkl, g)
        return (q * d).sum((-1, -2))
    # move Gamma_kl onto P_n: its free index becomes the partner's
    n = torch.einsum("kl,xnlcf->xnkcf" if sn == "l" else "lk,xnlcf->xnkcf", gkl, n)
    return torch.einsum("xnkcf,xnkcf->x", n, g if si == "n" else g.transpose(1, 2))


def _sums(site, latt):
    return site.reshape(site.shape[:-1] + (2, latt[3], -1)).sum((-1, -3))


def _exact_baryon(props, types, gij, gkl, ws):
    """[len(types), len(ws), V]."""
    v = len(props[0])
    out = torch.empty((len(types), len(ws), v), dtype=torch.complex128, device=DEVICE)
    for s in _chunks(v):
        pi, pj, pn = (q[s].to(torch.complex128) for q in props)
        g = _open_diquark(pi, pj, gij)
        for a, t in enumerate(types):
            for b, w in enumerate(ws):
                out[a, b, s] = _baryon_site(g, pn, t, gkl, w)
    return out


def _exact_sequential(props, t, slot, gij, gkl, w):
    """dC/dP_slot, with Gamma_ij moved onto P_j, W onto P_n and Gamma_kl onto the field that carries index l."""
    si, sj, sn = TYPES[t]
    q = [p.to(torch.complex128) for p in props]
    sides = [("i", si), ("i", sj), ("n", sn)]  # after the moves: P_j's first index is i, P_n's is n
    first = [None, gij, w]
    new = []
    for k in range(3):
        x = q[k]
        if first[k] is not None:
            x = torch.einsum("ab,xbtcf->xatcf", first[k], x)
        if sides[k][1] == "l":
            x = torch.einsum("kl,xalcf->xakcf", gkl, x)
        new.append(x)
    names = [a + b.replace("l", "k") for a, b in sides]
    u, v = [k for k in range(3) if k != slot]
    form = f"x{names[u]},x{names[v]}->x{names[slot]}"
    if names[slot] == "nn":  # the loop closed by Gamma_mn: a multiple of the identity
        d = _wedge(lambda a, b: torch.einsum(f"x{names[u]},x{names[v]}->x", a, b), new[u], new[v], (len(q[0]), 3, 3))
        d = torch.einsum("xcf,nt->xntcf", d, torch.eye(4, dtype=torch.complex128, device=DEVICE))
    elif "nn" in (names[u], names[v]):
        loop, other = (u, v) if names[u] == "nn" else (v, u)
        d = _wedge(lambda a, b: a[:, None, None] * b, torch.einsum("xnncf->xcf", new[loop]), new[other],
                   (len(q[0]), 4, 4, 3, 3))
    else:
        d = _wedge(lambda a, b: torch.einsum(form, a, b), new[u], new[v], (len(q[0]), 4, 4, 3, 3))
    if first[slot] is not None:
        d = torch.einsum("ab,xatcf->xbtcf", first[slot], d)
    if sides[slot][1] == "l":
        d = torch.einsum("kl,xakcf->xalcf", gkl, d)
    return d


def _products(pi, pj):
    """T[x][i][k][j][l] = sum over colours of P_i[i][k] conj(P_j[j][l])."""
    n = len(pi)
    return (pi.reshape(n, 16, 9) @ pj.reshape(n, 16, 9).mH).reshape(n, 4, 4, 4, 4)


def _pairs(t):
    """[.., 16, 16] of C_AB = sum (g5 A)[j][i] T[i][k][j][l] (g5 B)[k][l]."""
    gm = _gammas()
    g = _matrix(np.stack([gm[15] @ m for m in gm]))
    return torch.einsum("Aji,Bkl,...ikjl->...AB", g, g, t)


def _exact_momentum(props, latt, moms):
    """[momenta, Lt, 256]: the phase sum over each timeslice, direction by direction."""
    lx, ly, lz, lt = latt
    a, b = (p.reshape(2, lt, lz, ly, lx // 2, 144) for p in props)
    z, y, h = torch.meshgrid(*[torch.arange(n, device=DEVICE) for n in (lz, ly, lx // 2)], indexing="ij")
    nmax = int(np.abs(moms).max())
    n = torch.arange(-nmax, nmax + 1, device=DEVICE, dtype=torch.float64)

    def wave(length):
        arg = 2 * np.pi / length * (n[:, None] * torch.arange(length, device=DEVICE))
        return torch.complex(torch.cos(arg), torch.sin(arg))

    out = torch.empty((len(moms), lt, 256), dtype=torch.complex128, device=DEVICE)
    for t in range(lt):
        full = torch.empty((lz, ly, lx, 256), dtype=torch.complex128, device=DEVICE)
        for par in range(2):
            s = _products(a[par, t].reshape(-1, 16, 9).to(torch.complex128),
                          b[par, t].reshape(-1, 16, 9).to(torch.complex128))
            full[z.flatten(), y.flatten(), 2 * h.flatten() + ((par + t + z + y) & 1).flatten()] = s.reshape(-1, 256)
        s = torch.einsum("nx,zyxg->nzyg", wave(lx), full)
        s = torch.einsum("my,nzyg->mnzg", wave(ly), s)
        s = torch.einsum("lz,mnzg->lmng", wave(lz), s)
        out[:, t] = _pairs(s.reshape(-1, 4, 4, 4, 4)).reshape(-1, 256)
    return out


def exact(case, seed):
    op, latt = case["op"], _latt(case)
    gm = [_matrix(m) for m in _gammas()]
    if op == "batch":
        baryon, meson = [], []
        ws = [_matrix(w) for w in _projectors("both")]
        for lat, u, v, d in _sources(case, seed):
            baryon.append(_sums(_exact_baryon([u, v, d], range(6), gm[5], gm[5], ws), lat))
            meson.append(_exact_momentum([u, v], lat, _momenta(case["nmax"])))
        return {"baryon": baryon, "meson": meson}
    p = _props(case, seed)
    if op == "momentum":
        return _exact_momentum(p, latt, _momenta(case["nmax"]))
    if op in ("meson", "meson_all"):
        v = len(p[0])
        ga, every = case["gamma_a"], range(16)
        pick = [(ga, case["gamma_b"])] if op == "meson" else [(ga, g) if case["source"] else (g, ga) for g in every]
        out = torch.empty((len(pick), v), dtype=torch.complex128, device=DEVICE)
        for s in _chunks(v):
            t = _products(*(q[s].to(torch.complex128) for q in p))
            for k, (x, y) in enumerate(pick):
                out[k, s] = torch.einsum("ji,kl,xikjl->x", gm[15] @ gm[x], gm[15] @ gm[y], t)
        if op == "meson":
            return out[0]
        return _sums(out, latt) if case["summed"] else out
    ga, gb = gm[case["gamma_a"]], gm[case["gamma_b"]]
    if op == "diquark":
        sign = torch.tensor([1.0, 1.0, -1.0, -1.0], device=DEVICE, dtype=torch.float64)
        out = torch.empty((len(p[0]), 4, 4, 3, 3), dtype=torch.complex128, device=DEVICE)
        for s in _chunks(len(out)):
            g = _open_diquark(p[0][s].to(torch.complex128), p[1][s].to(torch.complex128), ga)
            d = torch.einsum("kl,xkmcf->xmlcf", gb, g).conj()
            out[s] = d * sign[:, None, None, None] * sign[:, None, None]
        return out
    if op == "sequential":
        out = torch.empty((len(p[0]), 4, 4, 3, 3), dtype=torch.complex128, device=DEVICE)
        for s in _chunks(len(out)):
            out[s] = _exact_sequential([q[s] for q in p], case["type"], case["slot"], ga, gb, gm[case["gamma_c"]])
        return out
    ws = [_matrix(w) for w in _projectors(case["proj"])]
    if op == "baryon_types":
        return list(_exact_baryon(p, range(6), ga, gb, ws)[:, 0])
    if op == "baryon":
        site = _exact_baryon(p, [case["type"]], ga, gb, ws)[0, 0]
        return _sums(site, latt) if case["summed"] else site
    return _sums(_exact_baryon(p, range(6), ga, gb, ws), latt)
