"""Builds at the sizes where the tile kernels' remainders change: basis sizes
off the 32-, 48-, 64- and 128-slot blocks, single and ragged tiles, both
precisions, against the CPU oracle (FP64 1e-10, INT8 1e-7)."""
import numpy as np
import pytest

import oracle as O
from pgxc import cases, lib

pytestmark = pytest.mark.gpu


def _case(natoms, lmax, functional, ispin=1, nang=26, nrad=9):
    c = cases.small_case(functional, seed=40 + natoms, natoms=natoms, nrad=nrad, nang=nang, nocc=max(2, natoms),
                         ispin=ispin, lmax=lmax)
    O.weight_case(c)
    return c


def _check(c, precision, threshold, tol):
    ref = O.xc_build(c)
    with lib.Context(c, precision=precision, screen_threshold=threshold) as ctx:
        ham, exc, nel = ctx.build()
    assert abs(exc - ref[1]) < tol and abs(nel - ref[2]) < tol
    assert float(np.max(np.abs(ham - ref[0]))) < tol


# nbas 22 .. 300: listed functions per tile on either side of each block size
@pytest.mark.parametrize("natoms,lmax", [(3, 0), (3, 1), (3, 2), (4, 2), (5, 3), (7, 2), (9, 3), (12, 2)])
def test_int8_block_remainders(natoms, lmax):
    _check(_case(natoms, lmax, "PBE"), "mixed", 1e-10, 1e-7)
