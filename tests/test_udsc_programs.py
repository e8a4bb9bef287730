"""The site programs of the table-driven baryons (udsc.site_program): merging
entries under exchange of equal flavours and choosing which blocks form a
diquark leaves every dataset's value unchanged.  Checked on the CPU against
the entries as they stand, and on the GPU at the edges of the kernel's tiles."""
import itertools

import numpy as np
import pytest

from plegma_b200 import udsc

EPS = np.zeros((3, 3, 3))
for p in itertools.permutations(range(3)):
    EPS[p] = round(np.linalg.det(np.eye(3)[list(p)]))
EPS2 = np.einsum("abc,xyz->axbycz", EPS, EPS).reshape(9, 9, 9)


def _triples(P):
    """eps eps' P1[b1] P2[b2] P3[b3] for all blocks."""
    return np.einsum("pqr,ip,jq,kr->ijk", EPS2, *P, optimize=True)


@pytest.mark.parametrize("flavours", ["uud", "udd", "uds", "uuu", "dsc", "ccc"])
def test_program_equals_the_entries(flavours):
    datasets = dict(udsc.products())[flavours]
    rng = np.random.default_rng(len(flavours) + ord(flavours[1]))
    props = {q: rng.standard_normal((16, 9)) + 1j * rng.standard_normal((16, 9)) for q in set(flavours)}
    full = _triples([props[q] for q in flavours])
    ref = np.array([sum(complex(w) * full[4 * t[0] + t[1], 4 * t[2] + t[3], 4 * t[4] + t[5]]
                        for t, w in zip(tuples, ws)) for _, tuples, ws in datasets])
    slots, warps = udsc.site_program(flavours, datasets)
    blocks = np.concatenate([props[q] for q in slots])
    full = _triples([blocks] * 3)
    got = np.zeros(len(datasets), dtype=complex)
    for groups in warps:
        for a, bs in groups:
            for b, dots in bs:
                for z, entries in dots:
                    for d, w in entries:
                        got[d] += w * full[a, b, z]
    # at most 2400 terms of up to 25 times the result: 2400 x 25 x 2^-53 < 1e-11
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    assert len(warps) == udsc.PROGRAM_WARPS


@pytest.mark.gpu
@pytest.mark.parametrize("L", [(1, 1, 1, 3), (3, 7, 3, 3), (4, 4, 2, 3), (11, 3, 1, 3)])  # 1, 63, 32, 33 sites
@pytest.mark.parametrize("split", [False, True])
def test_tile_edges_and_windows_per_flavour(L, split):
    """u holds all slices, d two of three: the products of u alone keep theirs
    and do not join the u,d launch, those of d do."""
    import torch
    from plegma_b200 import lib as p2
    from p2test import device_props
    import oracle_py as orc
    ctx = p2.Context(L)
    src = (0, 0, 0, 1)
    (u,) = device_props(ctx, [(31, 0)], t0=1)
    (d,) = device_props(ctx, [(31, 1)], t0=1, t_first=1, nt=2)
    moms = p2.mom_list(2)
    req = ctx.udsc_request(src, 3, 0, moms=moms, prop_u=0, prop_d=1,
                           mode=p2.P2_SPLIT_FP16 if split else p2.P2_PLAIN_FP64)
    names = p2.udsc_datasets(req)
    out = torch.zeros((len(names), 3, len(moms)), dtype=torch.complex128, device="cuda")
    req.out = out.data_ptr()
    ctx.contract_udsc([ctx.prop(u.data_ptr()), ctx.prop(d.data_ptr(), t_first=1, nt=2)], req)
    ctx.sync()
    got = out.cpu().numpy()
    hu = u.cpu().numpy().reshape(144, 3, ctx.V3)
    hd = np.zeros_like(hu)
    hd[:, 1:3] = d.cpu().numpy().reshape(144, 2, ctx.V3)
    off = 0
    for key, dss in udsc.products():
        if names[off:off + len(dss)] != [n for n, _, _ in dss]:
            continue
        taus = [0, 1, 2] if "d" not in key else [0, 1]  # global times 1, 2, 0
        props = [(hu if c == "u" else hd).reshape(144, -1) for c in key]
        ref, asum = orc.udsc_twopt(L, props, src, moms, dss, taus)
        g = got[off:off + len(dss)][:, taus].transpose(1, 0, 2)
        # FP32: a site's value is a sum of up to 2400 rounded products, 2^-24 each of terms
        # that reach 25 times the value; without an average over sites 3e-6 of sum |c| (test_gpu_split.py)
        tol = 1e-12 if not split else 1e-6 if ctx.V3 > 32 else 1e-5
        assert (np.abs(g - ref).max(axis=2) / np.maximum(asum, 1e-300)).max() < tol, key
        if "d" in key:
            assert not got[off:off + len(dss), 2].any()
        off += len(dss)
    assert off == len(names)
    ctx.close()
