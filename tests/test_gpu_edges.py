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


@pytest.mark.parametrize("functional,ispin", [("PBE", 1), ("VWN", 1), ("PBE", 2)])
@pytest.mark.parametrize("natoms,lmax", [(3, 0), (3, 1), (3, 2), (4, 2), (5, 3), (7, 2), (9, 3), (12, 2)])
def test_fp64_block_remainders(natoms, lmax, functional, ispin):
    _check(_case(natoms, lmax, functional, ispin), "fp64", 0.0, 1e-10)


# the symmetric half of the products: rho of an LDA and the tau sums and terms
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-7)])
@pytest.mark.parametrize("natoms,lmax", [(3, 1), (4, 2), (7, 2), (9, 3)])
def test_tau_block_remainders(natoms, lmax, precision, tol):
    _check(_case(natoms, lmax, "TPSS"), precision, 0.0, tol)


# a caller's P that is not symmetric: only its symmetric part counts, as in rho = phi^T P phi
def test_unsymmetric_density_matrix():
    c = _case(5, 3, "VWN")
    P = c.density_matrix()
    A = np.random.default_rng(3).normal(size=P.shape) * float(np.max(np.abs(P)))
    with lib.Context(c, screen_threshold=0.0) as ctx:
        ref, got = ctx.build_density(P), ctx.build_density(P + (A - A.transpose(0, 2, 1)))
    # rounding of sums of products up to max|A| rho-sized terms
    assert abs(got[1] - ref[1]) < 1e-9 and abs(got[2] - ref[2]) < 1e-9
    assert float(np.max(np.abs(got[0] - ref[0]))) < 1e-8
