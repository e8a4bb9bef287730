"""The axis-by-axis momentum projection (project_axes.cu) against the FP64
oracle's direct phase sum, at the edges of its rules: momenta at and beyond
L/2 (equal or opposite modulo L, no sine row), lists that are not closed under
sign flips, 1 to 9 rows per axis and the lists beyond it, fields of one
component and of more than a warp's 32, axes shorter and longer than a
128-byte chunk, a sub-lattice of a process grid.

Tolerance: a sum of n FP64 terms by another order differs by at most
n 2^-53 sum |f|; the transforms here have n <= 2000 and sum |f| <= 40 times
the largest result, so 1e-11 of the largest result bounds it."""
import numpy as np
import pytest
import torch

from plegma_b200 import lib as p2

import p2test  # noqa: F401  (puts the oracle on the path)
import oracle_py as orc

pytestmark = pytest.mark.gpu

ASYM = np.array([[0, 0, 0], [1, 0, 0], [-1, 2, 0], [0, -2, 1], [3, 1, -1], [5, -4, 2], [-3, 0, 7]], dtype=np.int32)


def _field(V3, dof, nt, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((dof, V3 * nt)) + 1j * rng.standard_normal((dof, V3 * nt))


@pytest.mark.parametrize("L,dof,moms", [
    ((4, 4, 4, 3), 1, p2.mom_list(9)),       # n = 2 is L/2, n = 3 is -1 mod 4
    ((3, 5, 2, 2), 33, ASYM),                # momenta beyond L/2, two components past a warp
    ((17, 3, 4, 2), 5, p2.mom_list(0)),      # one row
    ((9, 8, 7, 1), 70, p2.mom_list(16)),     # nine rows per axis, odd x axis of two chunks
    ((20, 6, 5, 2), 3, p2.mom_list(25)),     # |n| = 5: eleven rows, the direct sum
    ((1, 12, 6, 2), 32, p2.mom_list(4)),     # a single site along x
])
@pytest.mark.parametrize("sign", [1, -1])
def test_field_transform(L, dof, moms, sign):
    ctx = p2.Context(L)
    nt = L[3]
    f = _field(ctx.V3, dof, nt, 5)
    fd = torch.from_numpy(f).cuda()
    out = torch.full((nt, dof, len(moms)), complex(np.nan, np.nan), dtype=torch.complex128, device="cuda")
    for _ in range(2):  # tables built, tables kept
        ctx.ft_apply(fd.data_ptr(), dof, nt, moms, sign, out.data_ptr())
    ctx.sync()
    ref = orc.ft(L, f, dof, nt, moms, sign)
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()
    ctx.close()


def test_two_lists_and_signs_in_turn():
    ctx = p2.Context((6, 5, 4, 2))
    f = _field(ctx.V3, 4, 2, 6)
    fd = torch.from_numpy(f).cuda()
    for moms, sign in ((p2.mom_list(3), -1), (ASYM, 1), (p2.mom_list(3), 1), (p2.mom_list(2), -1)):
        out = torch.empty((2, 4, len(moms)), dtype=torch.complex128, device="cuda")
        ctx.ft_apply(fd.data_ptr(), 4, 2, moms, sign, out.data_ptr())
        ctx.sync()
        ref = orc.ft(ctx.L, f, 4, 2, moms, sign)
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()
    ctx.close()


def test_workspace_smaller_than_a_slice_and_sub_lattices():
    """One slice per chunk, and the sum over the halves of x and y gives the whole."""
    L, dof, moms = (8, 6, 4, 3), 7, p2.mom_list(5)
    f = _field(192, dof, 3, 7)
    ref = orc.ft(L, f, dof, 3, moms, -1)
    g = f.reshape(dof, 3, 4, 6, 8)
    got = 0
    for cx in range(2):
        for cy in range(2):
            ctx = p2.Context(L, procs=(2, 2, 1, 1), coords=(cx, cy, 0, 0))
            ctx.set_workspace(1)
            sub = torch.from_numpy(np.ascontiguousarray(g[:, :, :, 3 * cy:3 * cy + 3, 4 * cx:4 * cx + 4])).cuda()
            out = np.zeros((3, dof, len(moms)), dtype=np.complex128)
            ctx.ft_apply(sub.data_ptr(), dof, 3, moms, -1, out.ctypes.data, p2.P2_HOST)
            got = got + out
            ctx.close()
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
