"""Spin tables of the table-driven baryon two-point functions (the reference's
UDSC set: light, strange and charm octet/decuplet baryons with projected
interpolators), restated from the algorithm of the reference's generator
(python/baryons.py:27-543, output lib/kernels/PLEGMA_baryons_udsc_arrays.cuh).

Each baryon interpolator is J = sum_i k_i eps_abc (f1_a^T G_A f2_b) f3_c.  For
the correlator <J(x) Jbar(0)> with a projector P on the open spin of f3:
  1. list the six fields (three quarks with spin/colour slots 0..2, three
     antiquarks of Jbar = (f3bar, f1bar, f2bar) with slots 3..5);
  2. enumerate the Wick contractions (each quark paired with an antiquark of
     the same flavour; the sign is the parity of the pairing);
  3. move every contraction to the default view: propagators ordered by
     flavour (u, d, s, c), propagator k carrying spins (2k, 2k+1) and colours
     (k, 3+k); the colour relabelling multiplies the term by the parity of
     the colour permutation (the eps eps structure is fixed);
  4. for every non-zero (G_A[s0][s1], P[s2][s3], G_B[s4][s5]) the relabelled
     spin tuple collects value x coefficient;
  5. drop zeros and divide by the norm (sum k_i^2 for spin 1/2; 1/3, 1, 1/2
     for spin-3/2 sets of one, two, three flavour strings).
A site then contributes sum_entries w * sum_{eps eps'} P1[s0][s1][a][a']
P2[s2][s3][b][b'] P3[s4][s5][c][c'] (lib/kernels/PLEGMA_baryons_udsc.cu:85-134).

Weights are kept in single precision, as the reference's float2 tables are.
"""
from __future__ import annotations

import itertools
from typing import Dict, List, Tuple

import numpy as np

from . import spin

I = 1j
ONE = np.eye(4, dtype=complex)
GX, GY, GZ, GT = spin.G1, spin.G2, spin.G3, spin.G4
C = I * GY @ GT
G5 = GX @ GY @ GZ @ GT
CG5 = C @ G5
IGTCG5 = I * GT @ CG5
PP = 0.5 * (ONE + GT)
PM = 0.5 * (ONE - GT)
CGX, CGY, CGZ = C @ GX, C @ GY, C @ GZ

# interpolator sets: name -> list of (projector, G_A at the sink, G_B at the source)
SETS = {
    0.5: [
        ("Pp-Cg5-Cg5", [(PP, CG5, CG5)]),
        ("Pm-Cg5-Cg5", [(PM, CG5, CG5)]),
        ("Pp-igtCg5-igtCg5", [(PP, IGTCG5, IGTCG5)]),
        ("Pm-igtCg5-igtCg5", [(PM, IGTCG5, IGTCG5)]),
        ("g5Ppg5-C-C", [(G5 @ PP @ G5, C, C)]),
        ("g5Pmg5-C-C", [(G5 @ PM @ G5, C, C)]),
    ],
    1.5: [
        ("Pp-Cgi-Cgi", [(PP, CGX, CGX), (PP, CGY, CGY), (PP, CGZ, CGZ)]),
        ("Pm-Cgi-Cgi", [(PM, CGX, CGX), (PM, CGY, CGY), (PM, CGZ, CGZ)]),
        ("Ppgigj-Cgi-Cgj", [(PP @ GX @ GY, CGX, CGY), (PP @ GX @ GZ, CGX, CGZ), (PP @ GY @ GZ, CGY, CGZ),
                            (PP @ GY @ GX, CGY, CGX), (PP @ GZ @ GX, CGZ, CGX), (PP @ GZ @ GY, CGZ, CGY)]),
        ("Pmgigj-Cgi-Cgj", [(PM @ GX @ GY, CGX, CGY), (PM @ GX @ GZ, CGX, CGZ), (PM @ GY @ GZ, CGY, CGZ),
                            (PM @ GY @ GX, CGY, CGX), (PM @ GZ @ GX, CGZ, CGX), (PM @ GZ @ GY, CGZ, CGY)]),
    ],
}

# (name, flavour strings f1-f2-f3, coefficients, spin), in the reference's order
BARYONS: List[Tuple[str, List[str], List[int], float]] = [
    ("Xicc++", ["ch-up-ch"], [1], 0.5),
    ("Xicc+", ["ch-dn-ch"], [1], 0.5),
    ("Omegacc+", ["ch-sr-ch"], [1], 0.5),
    ("Sigmac++", ["up-ch-up"], [1], 0.5),
    ("Sigmac+", ["up-ch-dn", "dn-ch-up"], [1, 1], 0.5),
    ("Sigmac0", ["dn-ch-dn"], [1], 0.5),
    ("Xi'c+", ["up-ch-sr", "sr-ch-up"], [1, 1], 0.5),
    ("Xi'c0", ["dn-ch-sr", "sr-ch-dn"], [1, 1], 0.5),
    ("Omegac0", ["sr-ch-sr"], [1], 0.5),
    ("Lambdac+", ["up-dn-ch", "up-ch-dn", "dn-ch-up"], [2, 1, -1], 0.5),
    ("Xic+", ["sr-up-ch", "sr-ch-up", "up-ch-sr"], [2, 1, -1], 0.5),
    ("Xic0", ["sr-dn-ch", "sr-ch-dn", "dn-ch-sr"], [2, 1, -1], 0.5),
    ("proton", ["up-dn-up"], [1], 0.5),
    ("neutron", ["dn-up-dn"], [1], 0.5),
    ("Lambda", ["up-dn-sr", "up-sr-dn", "dn-sr-up"], [2, 1, -1], 0.5),
    ("Sigma+", ["up-sr-up"], [1], 0.5),
    ("Sigma0", ["up-sr-dn", "dn-sr-up"], [1, 1], 0.5),
    ("Sigma-", ["dn-sr-dn"], [1], 0.5),
    ("Xi0", ["sr-up-sr"], [1], 0.5),
    ("Xi-", ["sr-dn-sr"], [1], 0.5),
    ("Omegaccc++", ["ch-ch-ch"], [1], 1.5),
    ("Xi*cc++", ["ch-up-ch", "ch-ch-up"], [2, 1], 1.5),
    ("Xi*cc+", ["ch-dn-ch", "ch-ch-dn"], [2, 1], 1.5),
    ("Omega*cc+", ["ch-sr-ch", "ch-ch-sr"], [2, 1], 1.5),
    ("Sigma*c++", ["up-up-ch", "ch-up-up"], [1, 2], 1.5),
    ("Sigma*c+", ["up-dn-ch", "dn-ch-up", "ch-up-dn"], [1, 1, 1], 1.5),
    ("Sigma*c0", ["dn-dn-ch", "ch-dn-dn"], [1, 2], 1.5),
    ("Xi*c+", ["up-sr-ch", "sr-ch-up", "ch-up-sr"], [1, 1, 1], 1.5),
    ("Xi*c0", ["dn-sr-ch", "sr-ch-dn", "ch-dn-sr"], [1, 1, 1], 1.5),
    ("Omega*c0", ["sr-ch-sr", "sr-sr-ch"], [2, 1], 1.5),
    ("Delta++", ["up-up-up"], [1], 1.5),
    ("Delta+", ["up-dn-up", "up-up-dn"], [2, 1], 1.5),
    ("Delta0", ["dn-up-dn", "dn-dn-up"], [2, 1], 1.5),
    ("Delta-", ["dn-dn-dn"], [1], 1.5),
    ("Sigma*+", ["up-up-sr", "sr-up-up"], [1, 2], 1.5),
    ("Sigma*0", ["up-dn-sr", "dn-sr-up", "sr-up-dn"], [1, 1, 1], 1.5),
    ("Sigma*-", ["dn-dn-sr", "sr-dn-dn"], [1, 2], 1.5),
    ("Xi*0", ["sr-up-sr", "sr-sr-up"], [2, 1], 1.5),
    ("Xi*-", ["sr-dn-sr", "sr-sr-dn"], [2, 1], 1.5),
    ("Omega-", ["sr-sr-sr"], [1], 1.5),
]

FLAVOUR_ORDER = {"up": 0, "dn": 1, "sr": 2, "ch": 3}

# a field: (flavour, is_antiquark, slot); a propagator: (flavour, quark slot, antiquark slot)
Field = Tuple[str, bool, int]
Prop = Tuple[str, int, int]


def contractions(fields: List[Field]) -> List[Tuple[int, List[Prop]]]:
    """All Wick contractions of the fields as (sign, propagators).  The sign is
    the parity of bringing every (quark, antiquark) pair next to each other,
    quark first, taken pair by pair from the first field."""
    if not fields:
        return [(1, [])]
    head, rest = fields[0], fields[1:]
    out = []
    for i, f in enumerate(rest):
        if f[0] != head[0] or f[1] == head[1]:
            continue
        # moving f next to head crosses i fields; an antiquark-first pair flips once more
        sign = (-1) ** i * (1 if f[1] else -1)
        quark, anti = (head, f) if f[1] else (f, head)
        for s, props in contractions(rest[:i] + rest[i + 1:]):
            out.append((sign * s, [(quark[0], quark[2], anti[2])] + props))
    return out


def parity(perm: List[int]) -> int:
    p, seen = 1, [False] * len(perm)
    for i in range(len(perm)):
        if seen[i]:
            continue
        j, n = i, 0
        while not seen[j]:
            seen[j] = True
            j = perm[j]
            n += 1
        if n % 2 == 0:
            p = -p
    return p


def to_default_view(props: List[Prop]) -> Tuple[Dict[int, int], int]:
    """(spin slot map original -> default, colour sign) of one contraction.
    Default propagator k (flavour-sorted) has quark slot k and antiquark slot
    3 + k for colour, and spins 2k, 2k + 1."""
    flav = sorted((p[0] for p in props), key=lambda f: FLAVOUR_ORDER[f])
    free = list(range(3))
    spin_map, colour = {}, [0] * 6
    for fl, q, a in props:
        k = next(j for j in free if flav[j] == fl)
        free.remove(k)
        spin_map[q], spin_map[a] = 2 * k, 2 * k + 1
        colour[q], colour[a] = k, 3 + k
    return spin_map, parity(colour)


def nonzero_triples(mats):
    """(s0..s5, value) for the non-zero entries of the outer product of three 4x4 matrices."""
    nz = [[(r, c, m[r, c]) for r in range(4) for c in range(4) if abs(m[r, c]) > 1e-12] for m in mats]
    for (a, b, va), (c, d, vb), (e, f, vc) in itertools.product(*nz):
        yield (a, b, c, d, e, f), va * vb * vc


def baryon_tables(name, flavs, coeffs, spin_):
    """{set name: {6-tuple: weight}} and the flavour key of one baryon."""
    terms = []  # (coefficient, spin map)
    for fj, kj in zip(flavs, coeffs):
        q = fj.split("-")
        for fb, kb in zip(flavs, coeffs):
            qb = fb.split("-")
            fields = [(q[0], False, 0), (q[1], False, 1), (q[2], False, 2),
                      (qb[2], True, 3), (qb[0], True, 4), (qb[1], True, 5)]
            for s, props in contractions(fields):
                smap, csign = to_default_view(props)
                terms.append((kj * kb * s * csign, smap))
    if spin_ == 0.5:
        norm = float(sum(k * k for k in coeffs))
    else:
        norm = {3: 0.5, 2: 1.0, 1: 1.0 / 3.0}[len(coeffs)]
    out = {}
    for set_name, triples in SETS[spin_]:
        acc: Dict[Tuple[int, ...], complex] = {}
        for proj, ga, gb in triples:
            nz = list(nonzero_triples([ga, proj, gb]))
            for k, smap in terms:
                for tup, v in nz:
                    new = [0] * 6
                    for src, dst in smap.items():
                        new[dst] = tup[src]
                    key = tuple(new)
                    acc[key] = acc.get(key, 0) + v * k
        out[set_name] = {key: v / norm for key, v in acc.items() if not np.isclose(v, 0)}
    flav0 = sorted(flavs[0].split("-"), key=lambda f: FLAVOUR_ORDER[f])
    return out, "".join(f[0] for f in flav0)


def dataset_name(baryon: str, set_name: str) -> str:
    for a, b in (("+", "Pl"), ("-", "Mn"), ("*", "St"), ("'", "Pr")):
        baryon = baryon.replace(a, b)
    return baryon + "/" + set_name.replace("-", "_")


def products():
    """[(product 'uud', [(dataset name, [(s0..s5)], [complex64 weight])])] in the
    reference's product and dataset order."""
    prods: Dict[str, list] = {}
    for name, flavs, coeffs, sp in BARYONS:
        sets, key = baryon_tables(name, flavs, coeffs, sp)
        lst = prods.setdefault(key, [])
        for set_name, _ in SETS[sp]:
            ent = sets[set_name]
            lst.append((dataset_name(name, set_name), list(ent.keys()),
                        [np.complex64(v) for v in ent.values()]))
    return list(prods.items())


def names_digest(names) -> str:
    import hashlib
    return hashlib.sha256("\n".join(names).encode()).hexdigest()[:16]


def ordered_digest(idx, vals) -> str:
    """Digest of one dataset in entry order: (6 indices, weight rounded to single precision)."""
    import hashlib
    rows = [(tuple(int(x) for x in t), float(np.float32(np.real(v))) + 0.0, float(np.float32(np.imag(v))) + 0.0)
            for t, v in zip(idx, vals)]
    return hashlib.sha256(repr(rows).encode()).hexdigest()[:16]


def table_digest(idx, vals) -> str:
    """Order-independent digest of one dataset: sorted (tuple, weight rounded to 6 digits)."""
    import hashlib
    rows = sorted((tuple(int(x) for x in t), round(float(np.real(v)), 6) + 0.0, round(float(np.imag(v)), 6) + 0.0)
                  for t, v in zip(idx, vals))
    return hashlib.sha256(repr(rows).encode()).hexdigest()[:16]


#: Warps that share a site program (udsc.cu)
PROGRAM_WARPS = 8


def site_program(flavours, datasets):
    """Contraction program of one flavour product, see udsc.cu.

    Every term w eps eps' P1[b1] P2[b2] P3[b3] (b = spin block) is symmetric
    under exchange of equal flavours together with their blocks, so terms that
    differ by such an exchange are merged and each distinct triple of
    (flavour, block) is evaluated once for all datasets.  A triple is a
    diquark of two of its members dotted with the third; the diquarks are a
    greedy cover of the triples (each covers as many of those left as any
    other), so few of them are built.

    Returns (distinct flavours, per-warp lists of
    (A, [(B, [(Z, [(dataset, weight)])])])): the diquark of blocks A and B, its
    dots with blocks Z, and what each dot adds to the datasets; block
    16 slot + b, slot the index among the distinct flavours."""
    slots = sorted(set(flavours), key="udsc".index)
    weights: Dict[tuple, Dict[int, float]] = {}
    for d, (_, tuples, ws) in enumerate(datasets):
        for t, w in zip(tuples, ws):
            if abs(np.imag(w)) > 1e-12:
                raise ValueError("complex table weight")
            key = tuple(sorted(16 * slots.index(f) + 4 * t[2 * i] + t[2 * i + 1] for i, f in enumerate(flavours)))
            row = weights.setdefault(key, {})
            row[d] = row.get(d, 0.0) + float(np.real(w))
    triples = [k for k, row in weights.items() if any(abs(w) > 1e-9 for w in row.values())]
    # greedy cover: pairs of each triple, with the triples left to cover
    def pairs(t):
        return {(t[0], t[1]), (t[0], t[2]), (t[1], t[2])}

    def third(t, p):
        rest = list(t)
        for b in p:
            rest.remove(b)
        return rest[0]
    left: Dict[tuple, set] = {}
    for t in triples:
        for p in pairs(t):
            left.setdefault(p, set()).add(t)
    cover: Dict[tuple, list] = {}
    while any(left.values()):
        best = max(sorted(left), key=lambda p: len(left[p]))
        cover[best] = sorted(left[best])
        for t in cover[best]:
            for p in pairs(t):
                left[p].discard(t)
    # pairs that share a block become neighbours, so a warp loads that block once
    degree: Dict[int, int] = {}
    for p in cover:
        for b in set(p):
            degree[b] = degree.get(b, 0) + 1
    steps = []
    for p, ts in cover.items():
        a, b = p if degree[p[0]] >= degree[p[1]] else (p[1], p[0])
        dots = [(third(t, p), sorted((d, w) for d, w in weights[t].items() if abs(w) > 1e-9)) for t in ts]
        steps.append((a, b, dots))
    steps.sort(key=lambda q: (q[0], q[1]))
    cost = [36 + sum(9 + 2 * len(e) for _, e in dots) for _, _, dots in steps]
    # contiguous ranges of equal cost (smallest largest range, by bisection)
    def ranges(limit):
        out, acc = [[]], 0
        for i, c in enumerate(cost):
            if acc + c > limit and out[-1]:
                out.append([])
                acc = 0
            out[-1].append(i)
            acc += c
        return out
    lo, hi = max(cost), sum(cost)
    while lo < hi:
        mid = (lo + hi) // 2
        if len(ranges(mid)) <= PROGRAM_WARPS:
            hi = mid
        else:
            lo = mid + 1
    parts = ranges(lo)
    parts += [[] for _ in range(PROGRAM_WARPS - len(parts))]
    warps = []
    for part in parts:
        groups: List[tuple] = []
        for i in part:
            a, b, dots = steps[i]
            if not groups or groups[-1][0] != a:
                groups.append((a, []))
            groups[-1][1].append((b, dots))
        warps.append(groups)
    return slots, warps


#: Record types of an encoded program
REC_A, REC_B, REC_DOT, REC_END = range(4)


def encode_programs(prods):
    """(records, weights, program of each product, [(datasets, first record of each warp)], cases): the
    site programs as one stream of 32-bit records, equal programs stored once.  A record is
    type | block << 2 | case << 8 | weights << 16.  REC_A: the block becomes A; REC_B: it makes the
    diquark with A; REC_DOT: its dot with the diquark, times weights[weights + i], is added to dataset
    i of the case.  cases[0] and cases[1] are the lists of datasets (tuples) that the dots of programs
    of up to ten datasets, and of more, contribute to."""
    code: List[int] = []
    rows: Dict[tuple, int] = {}
    values: List[float] = []
    programs, which, seen = [], [], {}
    cases: Tuple[List[tuple], List[tuple]] = ([], [])

    def record(kind, block, case=0, first=0):
        code.append(kind | block << 2 | case << 8 | first << 16)
    for flavours, datasets in prods:
        _, warps = site_program(flavours, datasets)
        ident = repr(warps)
        if ident not in seen:
            starts = []
            mine = cases[0 if len(datasets) <= 10 else 1]
            for groups in warps:
                starts.append(len(code))
                for a, bs in groups:
                    record(REC_A, a)
                    for b, dots in bs:
                        record(REC_B, b)
                        for block, entries in dots:
                            support, row = tuple(d for d, _ in entries), tuple(w for _, w in entries)
                            if support not in mine:
                                mine.append(support)
                            if row not in rows:
                                rows[row] = len(values)
                                values.extend(row)
                            record(REC_DOT, block, mine.index(support), rows[row])
                record(REC_END, 0)
            seen[ident] = len(programs)
            programs.append((len(datasets), starts))
        which.append(seen[ident])
    for _ in range(2):  # a warp reads two records ahead
        record(REC_END, 0)
    if len(values) >= 1 << 16 or max(len(c) for c in cases) > 256 or max(n for n, _ in programs) > 16:
        raise ValueError("site program does not fit its encoding")
    return code, values, which, programs, cases


def emit_header(path: str) -> bool:
    """C header with the tables (generated at build time); True if the file changed."""
    prods = products()
    names, ds_begin, pflav = [], [0], []
    for key, dss in prods:
        pflav.append(key)
        names += [name for name, _, _ in dss]
        ds_begin.append(len(names))
    L = ["// Generated by plegma_b200/udsc.py: table-driven baryon spin tables.", "#pragma once", "",
         f"constexpr int kUdscProducts = {len(prods)};",
         f"constexpr int kUdscDatasets = {len(names)};",
         "static const char kUdscProduct[kUdscProducts][4] = {" + ", ".join(f'"{k}"' for k in pflav) + "};",
         "static const int kUdscDsBegin[kUdscProducts + 1] = {" + ", ".join(map(str, ds_begin)) + "};",
         "static const char* const kUdscName[kUdscDatasets] = {" + ", ".join(f'"{n}"' for n in names) + "};"]
    code, values, which, programs, cases = encode_programs(prods)
    L += ["", f"constexpr int kUdscWarps = {PROGRAM_WARPS};",
          "static const int kUdscProgram[kUdscProducts] = {" + ", ".join(map(str, which)) + "};",
          f"static const int kUdscProgramStart[{len(programs)}][kUdscWarps] = {{" +
          ", ".join("{" + ", ".join(map(str, st)) + "}" for _, st in programs) + "};",
          f"constexpr int kUdscCodeWords = {len(code)};",
          "#define P2_INIT_UDSC_CODE {" + ",".join("%du" % w for w in code) + "}",
          f"constexpr int kUdscWeights = {len(values)};",
          "#define P2_INIT_UDSC_WEIGHTS {" + ",".join("%.17g" % v for v in values) + "}"]
    # switch bodies: P2_ADD(d, i) adds weight i times the dot to dataset d
    for name, lists in zip(("10", "16"), cases):
        L.append(f"#define P2_UDSC_CASES_{name} " + " ".join(
            f"case {i}: " + " ".join(f"P2_ADD({d}, {k})" for k, d in enumerate(ds)) + " break;"
            for i, ds in enumerate(lists)))
    text = "\n".join(L) + "\n"
    try:
        with open(path) as f:
            if f.read() == text:
                return False
    except FileNotFoundError:
        pass
    with open(path, "w") as f:
        f.write(text)
    return True
