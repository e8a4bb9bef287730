"""The contraction fused with the sums over x (contract_site*.cu) and its
dispatch, both forms: every combination of blocks that takes it, shares a
request with blocks that go through the position buffer, or falls back, against
the FP64 oracle; rows shorter and longer than a tile of 32 (split) or 16 sites,
units of several rows, FP32 propagators.  Tolerance, relative to sum_x
|c_k(x,t)|: split err(t) <= 1e-6 (test_gpu_split.py) on lattices of enough
sites for the per-site rounding to average, plain 1e-13 (test_gpu_axes.py)."""
import numpy as np
import pytest
import torch

from plegma_b200 import lib as p2

from p2test import device_props, oracle_blocks, per_t_error, run

pytestmark = pytest.mark.gpu

SPLIT = p2.P2_SPLIT_FP16
FORMS = [(SPLIT, 1e-6), (p2.P2_PLAIN_FP64, 1e-13)]
D = p2.DELTA_ISO12 | p2.DELTA_ISO32
NUC, G16 = p2.NUCLEON_CG5, p2.MESON_G16


@pytest.mark.parametrize("what", [
    NUC, G16, NUC | G16, p2.DELTA_ISO12, p2.DELTA_ISO32, NUC | D | G16,
    NUC | D | G16 | p2.NUCLEON_NTOR,       # the second pass through the position buffer
    NUC | D | G16 | p2.MESON_ALL34,        # the first
    NUC | p2.NUCLEON_RTOR | p2.DELTA_ISO12 | p2.MESON_DIAG10,
])
@pytest.mark.parametrize("L", [(4, 6, 5, 4), (9, 4, 5, 3), (24, 2, 3, 3), (1, 10, 12, 3)])
@pytest.mark.parametrize("mode,tol", FORMS)
def test_blocks_and_row_lengths(what, L, mode, tol):
    ctx = p2.Context(L)
    src = (L[0] - 1, 1, 2, 1)
    bufs = device_props(ctx, [(61, 0), (61, 1)], t0=1)
    out, moms = run(ctx, bufs, src, L[3], what, q2max=4, mode=mode)
    taus = list(range(L[3]))
    ref = oracle_blocks(ctx.L, bufs, src, moms, what, taus)
    assert per_t_error(out, what, L[3], moms, ref, taus).max() < tol
    ctx.close()


@pytest.mark.parametrize("q2", [0, 9, 16, 25])  # 1, 7, 9 phase rows; eleven: through the position buffer
@pytest.mark.parametrize("fp32,mode,tol", [(True, SPLIT, 1e-6)] + [(False, *f) for f in FORMS])
def test_phase_rows_and_precisions(q2, fp32, mode, tol):
    ctx = p2.Context((13, 6, 5, 3))
    what = NUC | D | G16
    prec = p2.P2_FP32 if fp32 else p2.P2_FP64
    bufs = device_props(ctx, [(62, 0), (62, 1)], t0=0, precision=prec)
    out, moms = run(ctx, bufs, (5, 3, 1, 2), 3, what, q2max=q2, mode=mode, precision=prec)
    ref = oracle_blocks(ctx.L, bufs, (5, 3, 1, 2), moms, what, [0, 1, 2], fp32=fp32)
    assert per_t_error(out, what, 3, moms, ref, [0, 1, 2]).max() < tol
    ctx.close()


@pytest.mark.parametrize("mode", [m for m, _ in FORMS])
def test_rows_do_not_depend_on_the_batch(mode):
    """A slice's result is the same bits alone, in a chunk of slices and with one slice per chunk."""
    ctx = p2.Context((10, 7, 6, 5))
    what = NUC | D | G16
    bufs = device_props(ctx, [(63, 0), (63, 1)], t0=2)
    ref, moms = run(ctx, bufs, (1, 2, 3, 2), 5, what, q2max=5, mode=mode)
    ctx.set_workspace(1)
    got, _ = run(ctx, bufs, (1, 2, 3, 2), 5, what, q2max=5, mode=mode)
    assert np.array_equal(ref, got)
    one, _ = run(ctx, bufs, (1, 2, 3, 2), 1, what, q2max=5, mode=mode)
    a, b = p2.result_blocks(what, 5, len(moms), ref), p2.result_blocks(what, 1, len(moms), one)
    for bit in a:
        assert np.array_equal(a[bit][:, :, :1], b[bit])
    ctx.close()


def _constant_props(ctx, baryons, seed):
    """u and d without a dependence on the site (a free field from a wall
    source at p = 0) whose contractions are exact in FP32: one spin block each,
    integers of 7 bits on the colour diagonal (three-quark sums of at most 24
    bits) or of 12 bits in one colour entry (products of 24 bits)."""
    T = ctx.Ll[3]
    g = torch.Generator().manual_seed(seed)
    bufs = []
    for block in (0, 5):
        p = torch.zeros((144, T, ctx.V3), dtype=torch.complex128, device="cuda")
        for c in ((0, 4, 8) if baryons else (0,)):
            v = torch.randint(65, 128, (T,), generator=g) if baryons else torch.randint(2049, 4096, (T,), generator=g)
            p[9 * block + c] = v.cuda()[:, None]
        bufs.append(p)
    return bufs


@pytest.mark.parametrize("what,baryons", [
    (G16, False), (p2.MESON_ALL34 | p2.MESON_NEW10, False),         # sums over x in the contraction; from the position buffer
    (NUC | D, True), (NUC | p2.MESON_ALL34, True),
    ("udsc", True),
])
@pytest.mark.parametrize("L", [(64, 64, 1, 16), (128, 128, 1, 4), (236, 230, 1, 2)])
def test_sums_of_equal_values(what, baryons, L):
    """Adding one value again and again rounds the same way at every step, so
    the FP32 sums of the split form lose the most here (one running sum over x,
    then one over y: 1.7e-6 at 64 x 64, 7e-6 at 240 x 240).  Bound of the form:
    1e-6 of sum_x |c_k(x)|, which is |C(p = 0)| for equal values."""
    ctx = p2.Context(L)
    bufs = _constant_props(ctx, baryons, 64)
    T, moms = L[3], p2.mom_list(1)
    got = []
    for mode in (p2.P2_PLAIN_FP64, SPLIT):
        if what == "udsc":
            n = len(p2.udsc_datasets(ctx.udsc_request((0, 0, 0, 0), T, None, moms=moms, prop_u=0, prop_d=1)))
            out = torch.zeros(n * T * len(moms), dtype=torch.complex128, device="cuda")
            req = ctx.udsc_request((0, 0, 0, 0), T, out.data_ptr(), moms=moms, mode=mode, prop_u=0, prop_d=1)
            ctx.contract_udsc([ctx.prop(b.data_ptr()) for b in bufs], req)
            ctx.sync()
            got.append([out.cpu().numpy().reshape(n, T, len(moms))])
        else:
            out, _ = run(ctx, bufs, (0, 0, 0, 0), T, what, moms=moms, mode=mode)
            got.append([b for b in p2.result_blocks(what, T, len(moms), out).values()])
    for ref, res in zip(*got):
        ax = 2 if what == "udsc" else 3
        scale = np.abs(np.take(ref, [0], axis=ax))  # momentum 0 is p = 0
        held = scale > 1e-3 * scale.max()
        assert held.any()
        err = np.abs(res - ref) / np.where(held, scale, np.inf)
        assert err.max() < 1e-6, err.max()
    ctx.close()


@pytest.mark.parametrize("what,mode", [
    (NUC | D | G16, SPLIT), (NUC | D | G16, p2.P2_PLAIN_FP64),
    (p2.NUCLEON_NTOR | p2.NUCLEON_RTON | D | p2.MESON_ALL34, SPLIT),
    (p2.NUCLEON_NTOR | p2.NUCLEON_RTON | D | p2.MESON_ALL34, p2.P2_PLAIN_FP64),
    ("udsc", p2.P2_PLAIN_FP64),
])
def test_scratch_stays_within_the_workspace(what, mode):
    """The position buffer and the sums over x and y share the workspace
    budget: on a short x axis the sums take more than the buffer.  Same bits
    with and without the limit."""
    L, moms, T = (2, 64, 32, 24), p2.mom_list(1), 24
    budget, slack = 80 << 20, 12 << 20  # slack: tables, descriptors and the driver's granularity
    got = []
    for limit in (None, budget):  # the first pass loads the kernels and fills torch's pool
        torch.cuda.synchronize()
        ctx = p2.Context(L)
        bufs = device_props(ctx, [(67, 0), (67, 1)], t0=0)
        n = 28 if what == "udsc" else p2.components(what)
        out = torch.zeros(n * T * len(moms), dtype=torch.complex128, device="cuda")
        if limit:
            ctx.set_workspace(limit)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        props = [ctx.prop(b.data_ptr()) for b in bufs]
        if what == "udsc":
            ctx.contract_udsc(props, ctx.udsc_request((0, 0, 0, 0), T, out.data_ptr(), moms=moms, mode=mode, prop_u=0,
                                                      prop_d=1))
        else:
            ctx.contract_project(props, [ctx.request((0, 0, 0, 0), T, what, out.data_ptr(), mode=mode, moms=moms)])
        ctx.sync()
        used = free - torch.cuda.mem_get_info()[0]
        got.append(out.cpu().numpy())
        ctx.close()
    assert np.array_equal(got[0], got[1])
    assert used <= budget + slack, used >> 20


@pytest.mark.parametrize("L,what,q2,ran", [
    ((7, 40, 40, 9), NUC | G16, 2, "project_split_tc"),   # short x axis
    ((8, 40, 40, 9), NUC | G16, 2, "contract_site"),
    ((7, 40, 40, 8), NUC | G16, 2, "contract_site"),      # 89600 sites
    ((7, 40, 40, 9), NUC | G16, 10, "contract_site"),     # more than 128 momenta
    ((7, 40, 40, 9), G16 | p2.DELTA_ISO12, 2, "contract_site"),
    ((1, 50, 50, 4), G16, 2, "project_split_tc"),
    ((1, 50, 50, 3), G16, 2, "contract_site"),
    ((15, 30, 30, 8), p2.MESON_ALL34, 2, "project_split_tc"),
    ((16, 30, 30, 8), p2.MESON_ALL34, 2, "project_axis_x"),
    ((24, 25, 30, 12), NUC, 2, "project_axis_x"),         # the nucleon alone on a large lattice
    ((24, 25, 30, 11), NUC, 2, "contract_site"),
])
def test_split_dispatch_by_size(L, what, q2, ran):
    """Both sides of each line between the split form's paths: the kernel that runs and its result."""
    ctx = p2.Context(L)
    bufs = device_props(ctx, [(68, 0), (68, 1)], t0=0)
    ctx.profile()
    src = (L[0] - 1, 2, 3, 0)
    out, moms = run(ctx, bufs, src, 2, what, q2max=q2, mode=SPLIT)
    names = set(ctx.profile_read())
    assert ran in names and ("project_split_tc" in names) != ("project_axis_y" in names), names
    ref = oracle_blocks(ctx.L, bufs, src, moms, what, [1])
    assert per_t_error(out, what, 2, moms, ref, [1]).max() < 1e-6
    ctx.close()


@pytest.mark.parametrize("Lx,ran", [(3, "project_split_tc"), (4, "project_axis_x")])
def test_split_udsc_dispatch(Lx, ran):
    ctx = p2.Context((Lx, 60, 60, 10))
    bufs = device_props(ctx, [(69, 0), (69, 1)], t0=0)
    moms = p2.mom_list(2)
    got = []
    for mode in (p2.P2_PLAIN_FP64, SPLIT):
        out = torch.zeros(28 * len(moms), dtype=torch.complex128, device="cuda")
        ctx.profile()
        ctx.contract_udsc([ctx.prop(b.data_ptr()) for b in bufs],
                          ctx.udsc_request((0, 0, 0, 0), 1, out.data_ptr(), moms=moms, mode=mode, prop_u=0, prop_d=1))
        ctx.sync()
        got.append(out.cpu().numpy().reshape(28, len(moms)))
    assert ran in ctx.profile_read()
    # random signs: the values are about 1e-2 of sum_x |c|, which the form's 1e-6 is relative to
    assert np.abs(got[1] - got[0]).max() < 1e-4 * np.abs(got[0]).max()
    ctx.close()
