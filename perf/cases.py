"""The work that a program has the library do, as timed cases.

Every case goes through the public entry points (plegma_b200.lib, a thin
binding of the C ABI) on propagators that are resident on the GPU, as they
are after the solver.  Four kinds:

  twopt   contraction + momentum projection (p2_contract_project, or a
          recorded graph of it, or p2_contract_position): plain FP64 form and
          split form, FP64 and FP32 propagators, one source or a batch of
          sources with windows of their own, load-time transforms
  udsc    the table-driven u, d, s, c baryons (p2_contract_udsc), both forms
  ft      the momentum transform of a field (p2_ft_apply, p2_ft_apply_split)
  absorb  a propagator filled column by column from spinor fields, then
          rotated to the physical basis with the boundary sign
          (p2_prop_absorb, p2_prop_transform)

Propagator entries are complex Gaussians times exp(-decay |t - t0|), the
distribution of the library's benchmark configurations.  exact() states the
same quantities in plain torch in 64 bits.
"""
import functools
import itertools
import math
import random

import numpy as np
import torch

from plegma_b200 import lib as p2
from plegma_b200 import udsc

BITS = {"nucleon": p2.NUCLEON_CG5, "ntor": p2.NUCLEON_NTOR, "rton": p2.NUCLEON_RTON, "rtor": p2.NUCLEON_RTOR,
        "delta12": p2.DELTA_ISO12, "delta32": p2.DELTA_ISO32, "g16": p2.MESON_G16, "all34": p2.MESON_ALL34,
        "new10": p2.MESON_NEW10, "diag10": p2.MESON_DIAG10}
#: (groups, datasets, components) of each block of a result, in result order
SHAPE = {"nucleon": (1, 2, 16), "ntor": (1, 2, 16), "rton": (1, 2, 16), "rtor": (1, 2, 16), "delta12": (3, 2, 16),
         "delta32": (3, 2, 16), "g16": (1, 1, 256), "all34": (1, 1, 34), "new10": (1, 1, 10), "diag10": (1, 2, 10)}
#: complex products per site of each block with shared diquarks
PRODUCTS = {"nucleon": 3744, "ntor": 3744, "rton": 3744, "rtor": 3744, "delta12": 23400, "delta32": 18576,
            "g16": 2304, "all34": 2304, "new10": 2304, "diag10": 4608}
LIGHT = "nucleon+ntor+rton+rtor+delta12+delta32"
DIAG10 = [0, 5, 1, 2, 3, 4, 6, 7, 8, 9]


def listed():
    return [
        # the smallest call: one source on a tiny lattice, FP64; host calls and launches count
        dict(name="plain_4x8_nucleon", kind="twopt", lattice="4x4x4x8", windows="8", what="nucleon", q2=2,
             form="plain", precision="fp64", decay=0.5, transform=False, call="eager"),
        # a test-size lattice in the split form: still short kernels
        dict(name="split_8x16_nucleon_g16", kind="twopt", lattice="8x8x8x16", windows="16", what="nucleon+g16", q2=4,
             form="split", precision="fp64", decay=0.5, transform=False, call="eager"),
        # the plain form on a production lattice, all time slices of one source
        dict(name="plain_24x48_nucleon_g16", kind="twopt", lattice="24x24x24x48", windows="48", what="nucleon+g16",
             q2=9, form="plain", precision="fp64", decay=0.5, transform=False, call="eager"),
        # the split form on the benchmark's lattice, a window of 24 slices after the source
        dict(name="split_48x96_nucleon_g16", kind="twopt", lattice="48x48x48x96", windows="24", what="nucleon+g16",
             q2=9, form="split", precision="fp64", decay=0.5, transform=False, call="eager"),
        # a batch of sources with uneven windows and the Delta, replayed as one graph
        dict(name="batch_32x64_delta_graph", kind="twopt", lattice="32x32x32x64", windows="9,20,13,16",
             what="nucleon+delta12+delta32+g16", q2=9, form="split", precision="fp64", decay=0.5, transform=False,
             call="graph"),
        # propagators stored in FP32 on a large lattice, more momenta
        dict(name="fp32_64x128_delta", kind="twopt", lattice="64x64x64x128", windows="8",
             what="nucleon+delta12+delta32+g16", q2=16, form="split", precision="fp32", decay=0.4, transform=False,
             call="eager"),
        # the full light-baryon set and the diagonal mesons in FP64 on an odd lattice
        dict(name="plain_odd_light_diag10", kind="twopt", lattice="21x18x15x32", windows="16", what=LIGHT + "+diag10",
             q2=5, form="plain", precision="fp64", decay=0.5, transform=False, call="eager"),
        # the production driver on twisted-mass propagators: rotation and boundary sign on load, light baryons
        # and the meson lists of the reference's driver, zero and lowest momenta
        dict(name="split_24x48_rotated_light", kind="twopt", lattice="24x24x24x48", windows="24",
             what=LIGHT + "+all34+new10", q2=3, form="split", precision="fp64", decay=0.5, transform=True,
             call="eager"),
        # table-driven baryons of the u and d quarks in the split form
        dict(name="udsc_split_32x64_ud", kind="udsc", lattice="32x32x32x64", windows="16", quarks="ud", q2=9,
             form="split", precision="fp64", decay=0.5),
        # all 200 table-driven baryon datasets in FP64 on a small lattice
        dict(name="udsc_plain_16x32_udsc", kind="udsc", lattice="16x16x16x32", windows="16", quarks="udsc", q2=4,
             form="plain", precision="fp64", decay=0.5),
        # momentum transform of a position-space correlator field
        dict(name="ft_plain_24x48", kind="ft", lattice="24x24x24x48", dof=32, q2=9, sign=-1, form="plain"),
        # a propagator from twelve solver fields, rotated in place
        dict(name="absorb_24x48", kind="absorb", lattice="24x24x24x48", precision="fp64"),
    ]


def draw(rng):
    kind = rng.choice(["twopt", "twopt", "twopt", "twopt", "twopt", "udsc", "ft", "absorb"])

    def lattice(sites, window):
        v3 = max(8.0, sites / window)
        while True:
            side = v3 ** (1 / 3)
            ls = [max(2, min(64, round(side * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3)]
            if ls[0] * ls[1] * ls[2] <= 1.6 * v3:
                return ls

    form = rng.choice(["plain", "split", "split"])
    if kind == "twopt":
        what = rng.choice(["nucleon", "nucleon+g16", "nucleon+g16", "g16", "nucleon+delta12+delta32+g16", "delta12",
                           LIGHT + "+diag10", LIGHT + "+all34+new10", "nucleon+new10"])
        heavy = "delta" in what
        call = rng.choice(["eager", "eager", "eager", "graph", "position"])
        if call == "position":
            form = "plain"
        most = {("plain", True): 6e4, ("plain", False): 3e5, ("split", True): 4e5, ("split", False): 1e6}[form, heavy]
        if call == "position":
            most = 1e5
        sites = math.exp(rng.uniform(math.log(500), math.log(most)))
        window = rng.randint(1, 24)
        ls = lattice(sites, window)
        windows = [window] if call == "position" or rng.random() < 0.6 else [rng.randint(1, window) for _ in
                                                                             range(rng.randint(2, 5))]
        precision = "fp32" if form == "split" and rng.random() < 0.3 else "fp64"
        return dict(kind="twopt", lattice="x".join(map(str, ls + [window + rng.randint(0, 24)])),
                    windows=",".join(map(str, windows)), what=what, q2=rng.randint(0, 16), form=form,
                    precision=precision, decay=round(rng.uniform(0.2, 0.6), 2), transform=rng.random() < 0.2,
                    call=call)
    if kind == "udsc":
        quarks = rng.choice(["ud", "ud", "uds", "udsc"])
        most = {"ud": 2e5, "uds": 5e4, "udsc": 3e4}[quarks] * (1 if form == "plain" else 2)
        window = rng.randint(1, 20)
        ls = lattice(math.exp(rng.uniform(math.log(500), math.log(most))), window)
        return dict(kind="udsc", lattice="x".join(map(str, ls + [window + rng.randint(0, 24)])), windows=str(window),
                    quarks=quarks, q2=rng.randint(0, 12), form=form,
                    precision="fp32" if form == "split" and rng.random() < 0.3 else "fp64", decay=0.5)
    window = rng.randint(2, 48)
    if kind == "ft":
        dof = rng.choice([1, 2, 3, 10, 16, 20, 32, 34, 96])
        ls = lattice(math.exp(rng.uniform(math.log(2e3), math.log(2e7 / dof))), window)
        return dict(kind="ft", lattice="x".join(map(str, ls + [window])), dof=dof, q2=rng.randint(0, 16),
                    sign=rng.choice([-1, 1]), form=form)
    ls = lattice(math.exp(rng.uniform(math.log(2e3), math.log(6e5))), window)
    return dict(kind="absorb", lattice="x".join(map(str, ls + [window])), precision=rng.choice(["fp64", "fp32"]))


# ---- a program's state ---------------------------------------------------------

_stream = None


def _ctx(L):
    """A context on this program's stream: all its calls run there, one after the other."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    ctx = p2.Context(L)
    ctx.set_stream(_stream.cuda_stream)
    return ctx


def _lattice(case):
    return tuple(int(v) for v in case["lattice"].split("x"))


def _moms(q2):
    """Integer momenta of |n|^2 <= q2 by shells, each shell from the largest component down."""
    out = []
    for q in range(q2 + 1):
        r = math.isqrt(q)
        out += [(x, y, z) for x, y, z in itertools.product(range(r, -r - 1, -1), repeat=3) if x * x + y * y + z * z == q]
    return np.array(out, dtype=np.int32)


def _windows(case):
    return [int(v) for v in case["windows"].split(",")]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gaussian(shape, dtype, seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    t = torch.empty(shape, dtype=dtype, device=_device())
    torch.view_as_real(t).normal_(generator=g)
    return t


def _sources(case, seed):
    """A random source (x, y, z, t) of each window."""
    r = random.Random(seed)
    L = _lattice(case)
    return [tuple(r.randrange(L[d]) for d in range(4)) for _ in _windows(case)]


def _prop(case, seed, source, flavour):
    """[144][window][V3] of one source and flavour, the slices from the source's time on."""
    L = _lattice(case)
    n = _windows(case)[source]
    dtype = torch.complex64 if case["precision"] == "fp32" else torch.complex128
    u = _gaussian((144, n, L[0] * L[1] * L[2]), dtype, 1000 * seed + 10 * source + flavour)
    for j in range(n):
        u[:, j] *= math.exp(-case["decay"] * min(j, L[3] - j))
    return u


def _boundary(case):
    """Time below which the antiperiodic sign is applied."""
    return _lattice(case)[3] // 2


def prepare(case, seed):
    ctx = _ctx(_lattice(case))
    state = {"kind": case["kind"], "ctx": ctx}
    {"twopt": _prepare_twopt, "udsc": _prepare_udsc, "ft": _prepare_ft, "absorb": _prepare_absorb}[case["kind"]](
        case, seed, ctx, state)
    torch.cuda.synchronize()
    return state


def _prepare_twopt(case, seed, ctx, state):
    prec = p2.P2_FP32 if case["precision"] == "fp32" else p2.P2_FP64
    mode = p2.P2_SPLIT_FP16 if case["form"] == "split" else p2.P2_PLAIN_FP64
    what = sum(BITS[w] for w in case["what"].split("+"))
    moms = _moms(case["q2"])
    K = sum(math.prod(SHAPE[w]) for w in case["what"].split("+"))
    props, reqs, keep, outs = [], [], [], []
    for i, src in enumerate(_sources(case, seed)):
        n = _windows(case)[i]
        for f in range(2):
            u = _prop(case, seed, i, f)
            keep.append(u)
            xf = (p2.PROP_ROTATE_MINUS if f else p2.PROP_ROTATE_PLUS) | p2.PROP_BOUNDARY if case["transform"] else 0
            props.append(ctx.prop(u.data_ptr(), prec, t_first=src[3], nt=n, transform=xf, boundary_t0=_boundary(case)))
        cols = ctx.V3 if case["call"] == "position" else len(moms)
        out = torch.zeros(K * n * cols, dtype=torch.complex128, device="cuda")
        outs.append(out)
        reqs.append(ctx.request(src, n, what, out.data_ptr(), mode=mode, moms=moms, prop_u=2 * i, prop_d=2 * i + 1))
    torch.cuda.synchronize()  # the propagators are there before a graph's recording run reads them
    state.update(props=props, reqs=reqs, keep=keep, outs=outs, call=case["call"],
                 graph=ctx.graph(props, reqs) if case["call"] == "graph" else None)


def _prepare_udsc(case, seed, ctx, state):
    prec = p2.P2_FP32 if case["precision"] == "fp32" else p2.P2_FP64
    mode = p2.P2_SPLIT_FP16 if case["form"] == "split" else p2.P2_PLAIN_FP64
    src, n, moms = _sources(case, seed)[0], _windows(case)[0], _moms(case["q2"])
    keep = [_prop(case, seed, 0, f) for f in range(len(case["quarks"]))]
    props = [ctx.prop(u.data_ptr(), prec, t_first=src[3], nt=n) for u in keep]
    which = {"prop_" + q: i for i, q in enumerate(case["quarks"])}
    ndata = sum(len(d) for _, d in _products(case["quarks"]))
    out = torch.zeros(ndata * n * len(moms), dtype=torch.complex128, device="cuda")
    req = ctx.udsc_request(src, n, out.data_ptr(), moms=moms, mode=mode, **which)
    state.update(props=props, req=req, keep=keep, outs=[out])


def _ft_field(case, seed):
    L = _lattice(case)
    return _gaussian((case["dof"], L[3], L[0] * L[1] * L[2]), torch.complex128, 1000 * seed + 1)


def _prepare_ft(case, seed, ctx, state):
    L, moms = _lattice(case), _moms(case["q2"])
    out = torch.zeros(L[3] * case["dof"] * len(moms), dtype=torch.complex128, device="cuda")
    mode = p2.P2_SPLIT_FP16 if case["form"] == "split" else p2.P2_PLAIN_FP64
    state.update(field=_ft_field(case, seed), moms=moms, outs=[out], dof=case["dof"], nt=L[3], sign=case["sign"],
                 mode=mode)


def _vectors(case, seed):
    """[column nu 3 + c2][12][T V3] spinor fields."""
    L = _lattice(case)
    dtype = torch.complex64 if case["precision"] == "fp32" else torch.complex128
    return [_gaussian((12, L[0] * L[1] * L[2] * L[3]), dtype, 1000 * seed + c) for c in range(12)]


def _prepare_absorb(case, seed, ctx, state):
    vec = _vectors(case, seed)
    prop = torch.zeros((144, vec[0].shape[1]), dtype=vec[0].dtype, device="cuda")
    state.update(vec=vec, outs=[prop], t0=_boundary(case),
                 precision=p2.P2_FP32 if case["precision"] == "fp32" else p2.P2_FP64)


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "twopt":
        if state["call"] == "graph":
            state["graph"].launch()
        elif state["call"] == "position":
            ctx.contract_position(state["props"], state["reqs"][0])
        else:
            ctx.contract_project(state["props"], state["reqs"])
    elif state["kind"] == "udsc":
        ctx.contract_udsc(state["props"], state["req"])
    elif state["kind"] == "ft":
        ctx.ft_apply(state["field"].data_ptr(), state["dof"], state["nt"], state["moms"], state["sign"],
                     state["outs"][0].data_ptr(), mode=state["mode"])
    else:
        prop = state["outs"][0].data_ptr()
        for c, v in enumerate(state["vec"]):
            ctx.prop_absorb(prop, v.data_ptr(), c // 3, c % 3, state["precision"])
        ctx.prop_transform(prop, p2.PROP_ROTATE_PLUS | p2.PROP_BOUNDARY, state["t0"], state["precision"])
    return state["outs"]


# ---- what a pass cannot do without ----------------------------------------------

def _ft_products(q2, L):
    """Complex products per site and component of momentum sums taken one axis at a time."""
    m = _moms(q2)
    n1, n2 = len({v[0] for v in m.tolist()}), len({tuple(v[:2]) for v in m.tolist()})
    return n1 + n2 / L[0] + len(m) / (L[0] * L[1])


def work(case):
    L = _lattice(case)
    v3 = L[0] * L[1] * L[2]
    if case["kind"] == "absorb":
        n = 144 * v3 * L[3]
        return {"bytes": 2 * n * (8 if case["precision"] == "fp32" else 16), "flops": 4 * n}
    nmom = len(_moms(case["q2"]))
    if case["kind"] == "ft":
        n = case["dof"] * v3 * L[3]
        return {"bytes": 16 * n + 16 * case["dof"] * L[3] * nmom, "flops": 8 * n * _ft_products(case["q2"], L)}
    sites, slices = v3 * sum(_windows(case)), sum(_windows(case))
    esz = 8 if case["precision"] == "fp32" else 16
    if case["kind"] == "udsc":
        prods = _products(case["quarks"])
        K = sum(len(d) for _, d in prods)
        products = sum(36 * len({t[:4] for _, tups, _ in d for t in tups}) + 10 * sum(len(t) for _, t, _ in d)
                       for _, d in prods)
        read = len(case["quarks"]) * 144 * esz
    else:
        K = sum(math.prod(SHAPE[w]) for w in case["what"].split("+"))
        products = sum(PRODUCTS[w] for w in case["what"].split("+"))
        read = 2 * 144 * esz
        if case["call"] == "position":
            return {"bytes": sites * (read + 16 * K), "flops": 8 * sites * products}
    return {"bytes": sites * read + 16 * slices * K * nmom,
            "flops": 8 * sites * (products + K * _ft_products(case["q2"], L))}


def tolerance(case):
    if case["kind"] == "absorb":  # copies, one sum of four and a product: at most the last bit of each entry
        return {"rel": 2e-7 if case["precision"] == "fp32" else 1e-15}
    if case["form"] == "plain":  # 64-bit sums; against exact() up to 4e-15
        return {"rel": 3e-14}
    return {"rel": 5e-6}  # 32-bit site contraction and projection; against exact() up to 1.1e-6


# ---- the same quantities in plain torch, 64 bits ----------------------------------
# Dirac-Pauli basis: gamma_k = i [[0, sigma_k], [-sigma_k, 0]], gamma_4 = diag(1, 1, -1, -1),
# gamma_5 = gamma_1 gamma_2 gamma_3 gamma_4, C = i gamma_2 gamma_4.

_sigma = [np.array(m, dtype=complex) for m in ([[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]])]
_zero = np.zeros((2, 2))
GAMMA = [1j * np.block([[_zero, s], [-s, _zero]]) for s in _sigma] + [np.diag([1, 1, -1, -1]).astype(complex)]
G5 = GAMMA[0] @ GAMMA[1] @ GAMMA[2] @ GAMMA[3]
CMAT = 1j * GAMMA[1] @ GAMMA[3]
GAMMA16 = ([np.eye(4, dtype=complex)] + GAMMA + [G5] + [G5 @ g for g in GAMMA] +
           [-0.5j * (GAMMA[a] @ GAMMA[b] - GAMMA[b] @ GAMMA[a])
            for a, b in ((0, 1), (0, 2), (1, 2), (3, 0), (3, 1), (3, 2))])


def _bar(m):
    return GAMMA[3] @ m.conj().T @ GAMMA[3]


def _diquark(X, Y, gamma):
    """Q[s1][s2][c][e] = sum gamma[n][l] eps_abc eps_xye X[n][s1][a][x] Y[l][s2][b][y]."""
    Q = torch.zeros((4, 4, 3, 3, X.shape[-1]), dtype=torch.complex128, device=X.device)
    for n, l in zip(*np.nonzero(np.abs(gamma) > 1e-12)):
        x, y = X[n] * complex(gamma[n, l]), Y[l]
        for c, e in itertools.product(range(3), range(3)):
            a, b, p, q = (c + 1) % 3, (c + 2) % 3, (e + 1) % 3, (e + 2) % 3
            for (i, j), (k, m), s in (((a, b), (p, q), 1), ((a, b), (q, p), -1), ((b, a), (p, q), -1),
                                      ((b, a), (q, p), 1)):
                Q[:, :, c, e].add_(x[:, i, k][:, None] * y[:, j, m][None], alpha=s)
    return Q


def _wick(Q, Z, gbar, order):
    """T[m][r] of one Wick term: the lines of Q = Q^XY and Z end on the source spins named by `order`
    (n, l contracted with gbar[l][n], r open); the source's epsilon takes the colours in the order n, l, r."""
    sign = 1 if order in ("nlr", "lrn", "rnl") else -1
    T = 0
    if order[2] == "r":
        D = sum(complex(gbar[l, n]) * (Q[n, l] if order[0] == "n" else Q[l, n])
                for l, n in zip(*np.nonzero(np.abs(gbar) > 1e-12)))
        T = (D * Z).sum((2, 3))
    else:
        for l, n in zip(*np.nonzero(np.abs(gbar) > 1e-12)):
            at = {"l": l, "n": n}
            q = Q[:, at[order[1]]] if order[0] == "r" else Q[at[order[0]]]  # [r][c][e]
            T = T + complex(gbar[l, n]) * (q[None] * Z[:, at[order[2]]][:, None]).sum((2, 3))
    return sign * T


def _nucleon(A, B, sink, source):
    Q, g = _diquark(A, B, sink), _bar(source)
    return _wick(Q, A, g, "nlr") - _wick(Q, A, g, "rln")


def _spin(T, left, right):
    """left T right on [mu][mu'][V]."""
    l, r = (torch.as_tensor(m, device=T.device) for m in (left, right))
    return torch.einsum("ab,bcv,cd->adv", l, T, r)


def _block(name, U, D):
    """[group][dataset][component][V] of one block."""
    one = np.eye(4, dtype=complex)
    if name in ("nucleon", "ntor", "rton", "rtor"):
        sink = CMAT if name[0] == "r" else CMAT @ G5
        source = CMAT if name[-1] == "r" else CMAT @ G5
        left, right = (G5 if name[0] == "r" else one), (G5 if name[-1] == "r" else one)
        s = {"nucleon": 1, "ntor": -1, "rton": 1, "rtor": -1}[name]
        return torch.stack([s * _spin(_nucleon(A, B, sink, source), left, right).reshape(16, -1)
                            for A, B in ((U, D), (D, U))])[None]
    if name in ("delta12", "delta32"):
        out = []
        for k in range(3):
            cg = CMAT @ GAMMA[k]
            g = _bar(cg)
            row = []
            for A, B in ((U, D), (D, U)):
                aa = _diquark(A, A, cg)
                if name == "delta32":
                    T = (_wick(aa, A, g, "lrn") - _wick(aa, A, g, "rln") + _wick(aa, A, g, "rnl") -
                         _wick(aa, A, g, "nrl") - _wick(aa, A, g, "lnr") + _wick(aa, A, g, "nlr"))
                else:
                    ab = _diquark(A, B, cg)
                    T = (-4 * _wick(ab, A, g, "rln") + 2 * _wick(ab, A, g, "lrn") + 2 * _wick(aa, B, g, "rnl") -
                         2 * _wick(aa, B, g, "nrl") - 2 * _wick(ab, A, g, "nrl") - _wick(aa, B, g, "lnr") +
                         _wick(aa, B, g, "nlr") + 4 * _wick(ab, A, g, "nlr")) / 3
                row.append(T.reshape(16, -1))
            out.append(torch.stack(row))
        return torch.stack(out)
    if name == "diag10":
        return torch.stack([_mesons(A, A)[[17 * g for g in DIAG10]] for A in (U, D)])[None]
    m = _mesons(U, D)
    if name == "all34":
        m = m[[0, 5 * 17] + [16 * (i + 5 * h) + j + 5 * h for h in (0, 1) for i in range(1, 5) for j in range(1, 5)]]
    elif name == "new10":
        m = m[[17 * g for g in DIAG10]]
    return m[None, None]


def _mesons(A, B):
    """C[g1 16 + g2] = sum G1[d][a] A[a][b] G2[b][z] conj(B[d][z]) over spin and colour."""
    v = A.shape[-1]
    M = torch.einsum("icv,jcv->ijv", A.reshape(16, 9, v), B.reshape(16, 9, v).conj()).reshape(4, 4, 4, 4, v)
    G = torch.as_tensor(np.stack(GAMMA16), device=A.device)
    W = torch.einsum("gda,hbz->ghabdz", G, G).reshape(256, 256)
    return W @ M.reshape(256, v)


_tables = functools.lru_cache(udsc.products)


def _products(quarks):
    """Flavour products of the given quarks: the interpolator tables that the datasets are defined by."""
    return [(f, d) for f, d in _tables() if set(f) <= set(quarks)]


def _table_baryons(P, datasets):
    """[dataset][V]: sum w eps eps' P1[s0 s1] P2[s2 s3] P3[s4 s5]."""
    by_pair = {}
    for d, (_, tuples, weights) in enumerate(datasets):
        for t, w in zip(tuples, weights):
            W = by_pair.setdefault(tuple(t[:4]), np.zeros((len(datasets), 4, 4), dtype=complex))
            W[d, t[4], t[5]] += complex(w)
    z = P[2].reshape(16, 9, -1)
    out = torch.zeros((len(datasets), z.shape[-1]), dtype=torch.complex128, device=z.device)
    for (s0, s1, s2, s3), W in by_pair.items():
        x, y = P[0][s0, s1], P[1][s2, s3]
        q = []
        for c, e in itertools.product(range(3), range(3)):
            a, b, p, r = (c + 1) % 3, (c + 2) % 3, (e + 1) % 3, (e + 2) % 3
            q.append(x[a, p] * y[b, r] - x[a, r] * y[b, p] - x[b, p] * y[a, r] + x[b, r] * y[a, p])
        use = np.nonzero(np.abs(W).sum(axis=0).reshape(16))[0]
        dots = (torch.stack(q)[None] * z[torch.as_tensor(use, device=z.device)]).sum(1)
        out += torch.as_tensor(W.reshape(len(datasets), 16)[:, use], device=z.device) @ dots
    return out


def _phases(L, moms, origin, sign):
    """[momentum][V3] exp(sign i 2 pi n (x - origin) / L)."""
    m = torch.as_tensor(moms, dtype=torch.int64, device=_device())
    ph = None
    for d in (2, 1, 0):
        x = torch.arange(L[d], device=_device()) - origin[d]
        e = torch.remainder(m[:, d, None] * x[None], L[d]).double() * (2 * math.pi / L[d])
        e = torch.polar(torch.ones_like(e), sign * e)
        ph = e if ph is None else (ph[:, :, None] * e[:, None, :]).reshape(len(m), -1)
    return ph


def _transformed(P, flavour, sign):
    """Rotation to the physical basis (+ for the first flavour, - for the second), times the boundary sign."""
    s = 1j if flavour == 0 else -1j
    r = [2, 3, 0, 1]
    return sign * 0.5 * (P - P[r][:, r] + s * (P[:, r] + P[r]))


CHUNK = 16384  # sites at a time


def exact(case, seed):
    L = _lattice(case)
    v3 = L[0] * L[1] * L[2]
    if case["kind"] == "absorb":
        P = torch.stack([v.to(torch.complex128) for v in _vectors(case, seed)])  # [nu 3 + c2][mu 3 + c1][T V3]
        P = P.reshape(4, 3, 4, 3, L[3], v3).permute(2, 0, 3, 1, 4, 5)
        out = torch.empty((4, 4, 3, 3, L[3], v3), dtype=torch.complex128, device=P.device)
        for t in range(L[3]):
            out[..., t, :] = _transformed(P[..., t, :].contiguous(), 0, -1.0 if t < _boundary(case) else 1.0)
        return [out.reshape(144, -1)]
    moms = _moms(case["q2"])
    if case["kind"] == "ft":
        f, ph = _ft_field(case, seed), _phases(L, moms, (0, 0, 0), case["sign"])
        return [torch.stack([f[:, t] @ ph.T for t in range(L[3])]).reshape(-1)]
    outs = []
    for i, src in enumerate(_sources(case, seed)):
        n = _windows(case)[i]
        quarks = case["quarks"] if case["kind"] == "udsc" else "ud"
        props = {q: _prop(case, seed, i, f) for f, q in enumerate(quarks)}
        position = case.get("call") == "position"
        ph = None if position else _phases(L, moms, src, -1)
        parts = []  # per block: [group * dataset][tau][momentum or site][component]
        for t in range(n):
            sign = -1.0 if (src[3] + t) % L[3] < _boundary(case) else 1.0
            sums = None
            for x in range(0, v3, CHUNK):
                P = {q: u[:, t, x:x + CHUNK].to(torch.complex128).reshape(4, 4, 3, 3, -1) for q, u in props.items()}
                if case["kind"] == "udsc":
                    c = [_table_baryons([P[q] for q in f], d)[:, None] for f, d in _products(quarks)]
                else:
                    if case["transform"]:
                        P = {q: _transformed(v, f, sign) for f, (q, v) in enumerate(P.items())}
                    c = [_block(w, P["u"], P["d"]) for w in case["what"].split("+")]
                    c = [b.reshape(-1, b.shape[2], b.shape[3]) for b in c]
                if position:
                    got = c
                    sums = got if sums is None else [torch.cat((a, b), -1) for a, b in zip(sums, got)]
                else:
                    got = [b @ ph[:, x:x + CHUNK].T for b in c]
                    sums = got if sums is None else [a + b for a, b in zip(sums, got)]
            parts.append(sums)
        if position:  # [tau][component][site]
            outs.append(torch.stack([torch.cat([b.reshape(-1, v3) for b in p]) for p in parts]).reshape(-1))
        else:  # [group][dataset][tau][momentum][component] of every block
            outs.append(torch.cat([torch.stack([p[b] for p in parts], 1).transpose(2, 3).reshape(-1)
                                   for b in range(len(parts[0]))]))
    return outs
