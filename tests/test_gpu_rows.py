"""The contraction fused with the sums over x (contract_site*.cu) and its
dispatch, both forms: every combination of blocks that takes it, shares a
request with blocks that go through the position buffer, or falls back, against
the FP64 oracle; rows shorter and longer than a tile of 32 (split) or 16 sites,
units of several rows, FP32 propagators.  Tolerance, relative to sum_x
|c_k(x,t)|: split err(t) <= 1e-6 (test_gpu_split.py) on lattices of enough
sites for the per-site rounding to average, plain 1e-13 (test_gpu_axes.py)."""
import numpy as np
import pytest

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
