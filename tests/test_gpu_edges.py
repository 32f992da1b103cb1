"""Builds at the sizes where the tile kernels' remainders change: basis sizes
off the 32-, 48-, 64- and 128-slot blocks, single and ragged tiles, both
precisions, against the CPU oracle (FP64 1e-10, INT8 1e-7)."""
import ctypes as ct

import numpy as np
import pytest

import oracle as O
from pgxc import cases, lib

pytestmark = pytest.mark.gpu


def _case(natoms, lmax, functional, ispin=1, nang=26, nrad=9, nocc=None):
    c = cases.small_case(functional, seed=40 + natoms, natoms=natoms, nrad=nrad, nang=nang,
                         nocc=max(2, natoms) if nocc is None else nocc, ispin=ispin, lmax=lmax)
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


# 148 tiles (one per SM), a few more (even tile lists) and several per SM: INT8 against FP64
@pytest.mark.parametrize("functional", ["VWN", "PBE"])
@pytest.mark.parametrize("nrad,nang", [(24, 110), (25, 110), (40, 194)])
def test_int8_tile_lists(nrad, nang, functional):
    c = _case(7, 2, functional, nang=nang, nrad=nrad)
    r = []
    for precision in ("mixed", "fp64"):
        with lib.Context(c, precision=precision, screen_threshold=1e-10) as ctx:
            r.append(ctx.build())
    assert abs(r[0][1] - r[1][1]) < 1e-7 and abs(r[0][2] - r[1][2]) < 1e-7
    assert float(np.max(np.abs(r[0][0] - r[1][0]))) < 1e-7


# orbitals in the place of P, on either side of its 16-row stages and 64-column blocks and of the
# length where P is taken instead; occupations of both signs and none
@pytest.mark.parametrize("functional,ispin", [("VWN", 1), ("PBE", 1), ("PBE", 2), ("TPSS", 1), ("TPSS", 2)])
@pytest.mark.parametrize("nocc", [1, 15, 16, 17, 33, 64, 65, 100])
def test_fp64_orbital_remainders(nocc, functional, ispin):
    c = _case(12, 2, functional, ispin, nocc=nocc)
    c.occ[-1] *= -0.125
    c.occ[nocc // 2] = 0.0
    c.occ[0] = 2.0
    _check(c, "fp64", 0.0, 1e-10)


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


# the gradient on compact tiles: a shell with bare primitives only (not segmented), the most radial
# functions a shell may have, and the block sizes
def _wide(c, nrad):
    """The case's first shell replaced by nrad bare primitives."""
    ne, nc = int(c.shell_nexp[0]), int(c.shell_ncontr[0])
    e = np.exp(np.linspace(np.log(0.2), np.log(60.0), nrad))
    c.exponents = np.concatenate([e, c.exponents[ne:]])
    c.norms = np.concatenate([cases.primitive_norm(int(c.shell_l[0]), e), c.norms[ne:]])
    c.contractions = c.contractions[ne * nc:]
    for a, v in ((c.shell_nexp, nrad), (c.shell_nunc, nrad), (c.shell_ncontr, 0)):
        a[0] = v
    c.nbas += nrad - nc
    rng = np.random.default_rng(5)
    c.C = rng.normal(size=(c.nbas, c.nocc, c.ispin)) / c.nbas
    return c


@pytest.mark.parametrize("nrad,threshold", [(5, 0.0), (64, -1.0)])
@pytest.mark.parametrize("functional", ["VWN", "PBE"])
def test_gradient_of_unsegmented_shells(functional, nrad, threshold):
    c = _wide(cases.small_case(functional, seed=66, natoms=4, nrad=12, nang=50, nocc=5), nrad)
    ref, re = O.xc_gradient(c)
    with lib.Context(c, weighted=False, screen_threshold=threshold) as ctx:
        g, e = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref))))
    assert abs(e - re) < 1e-10 * max(1.0, abs(re))
    np.testing.assert_allclose(g, ref, rtol=0, atol=1e-10 * scale)


@pytest.mark.parametrize("natoms,lmax", [(3, 0), (5, 3), (9, 3), (12, 2)])
def test_gradient_block_remainders(natoms, lmax):
    c = cases.small_case("PBE", seed=40 + natoms, natoms=natoms, nrad=9, nang=26, nocc=max(2, natoms), lmax=lmax)
    ref, re = O.xc_gradient(c)
    with lib.Context(c, weighted=False, screen_threshold=1e-10) as ctx:
        g, e = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref))))
    assert abs(e - re) < 1e-10 * max(1.0, abs(re))
    np.testing.assert_allclose(g, ref, rtol=0, atol=1e-10 * scale)


# a caller whose number of orbitals creeps upwards: one staging buffer (with the padded buffers of
# every 16 orbitals, 2 ldc kpad doubles each, which a captured batch may hold: 13 MB), not one per step (72 MB)
def test_outgrown_orbital_buffers_are_released():
    import torch
    c = _case(16, 2, "VWN", nrad=6)
    rng = np.random.default_rng(8)
    C = rng.normal(size=(c.nbas, c.nbas, 1)) / c.nbas
    torch.cuda.init()
    with lib.Context(c, screen_threshold=0.0) as ctx:
        c.nocc = 1
        ctx.build(C=C[:, :1].T, occ=np.full(1, 2.0))
        free = torch.cuda.mem_get_info()[0]
        for c.nocc in range(2, c.nbas + 1):
            last = ctx.build(C=C[:, :c.nocc, 0].T, occ=np.full(c.nocc, 2.0))
        held = free - torch.cuda.mem_get_info()[0]
    steps = np.arange(16, c.nbas + 16, 16)
    assert held < 8 * (2 * (c.nbas + 64) * steps.sum() + (c.nbas + 1) * (c.nbas + 16)) + (8 << 20)
    with lib.Context(c, screen_threshold=0.0) as ctx:
        ref = ctx.build(C=C[:, :, 0].T, occ=np.full(c.nbas, 2.0))
    assert abs(last[1] - ref[1]) < 1e-10 and float(np.max(np.abs(last[0] - ref[0]))) < 1e-10


# a device wait that runs out (its error state set from the host, no wait is made to run out): the
# call reports it, the caller's outputs stay as they were, and the next call is whole again
def test_outputs_after_a_wait_that_ran_out():
    import torch
    from pgxc import abi
    c = _case(4, 2, "PBE")
    C, occ = torch.from_numpy(c.c_fortran()).cuda(), torch.from_numpy(c.occ_fortran()).cuda()
    ham = torch.full((c.xc_length,), 7.0, dtype=torch.float64, device="cuda")
    sums = torch.full((2,), 7.0, dtype=torch.float64, device="cuda")
    with lib.Context(c, precision="mixed", screen_threshold=1e-10) as ctx:
        ref = ctx.build()
        for call in (lambda: ctx.build_device(C.data_ptr(), occ.data_ptr(), ham.data_ptr(), sums.data_ptr()), ctx.build):
            assert lib.lib().pgxc_test_raise_wait_error(ctx.h) == 0
            with pytest.raises(lib.PgxcError) as e:
                call()
            assert e.value.status == abi.PGXC_ETIMEOUT
        torch.cuda.synchronize()
        assert bool((ham == 7.0).all()) and bool((sums == 7.0).all())
        ctx.build_device(C.data_ptr(), occ.data_ptr(), ham.data_ptr(), sums.data_ptr())
        assert abs(float(sums[0]) - ref[1]) < 1e-12
        assert float(np.max(np.abs(ham.cpu().numpy() - ref[0]))) < 1e-12


# psi of a larger grid (here 2,500 tiles x 48 orbitals, 120 MB) is held once a build by orbitals has been made, not
# by a context that is given density matrices; a build with more orbitals than there is room for makes more
def test_psi_is_made_by_the_builds_that_use_it():
    import torch
    c = _case(12, 2, "PBE", nrad=160, nang=194, nocc=40)
    P = c.density_matrix()
    torch.cuda.init()
    with lib.Context(c, screen_threshold=0.0) as ctx:
        ref = ctx.build_density(P)
        free = torch.cuda.mem_get_info()[0]
        c.nocc = 16
        ctx.build(C=c.C[:, :16, 0].T, occ=c.occ[:16, 0])
        few = free - torch.cuda.mem_get_info()[0]
        c.nocc = 40
        got = ctx.build()
        held = free - torch.cuda.mem_get_info()[0]
        tiles = ctx.screen_stats()["ntiles"]
    for orbitals, bytes_held in ((16, few), (48, held)):
        assert abs(bytes_held - orbitals * tiles * 1024) < 12 << 20  # (and the padded orbitals)
    assert abs(got[1] - ref[1]) < 1e-10 and abs(got[2] - ref[2]) < 1e-10
    assert float(np.max(np.abs(got[0] - ref[0]))) < 1e-10


# no room for psi (the rest of the device memory is taken): the build takes P; one that needs less is made by
# orbitals again once there is room
def test_builds_without_room_for_psi():
    import torch
    c = _case(12, 2, "PBE", nrad=160, nang=194, nocc=40)
    P = c.density_matrix()
    torch.cuda.init()
    with lib.Context(c, screen_threshold=0.0) as ctx:
        ref = ctx.build_density(P)
        tiles = ctx.screen_stats()["ntiles"]
        assert 48 * tiles * 1024 > 112 << 20
        torch.cuda.empty_cache()
        taken = torch.empty(torch.cuda.mem_get_info()[0] - (72 << 20), dtype=torch.uint8, device="cuda")
        got = ctx.build()
        del taken
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        c.nocc = 16
        ctx.build(C=c.C[:, :16, 0].T, occ=c.occ[:16, 0])
        held = free - torch.cuda.mem_get_info()[0]
    assert abs(got[1] - ref[1]) < 1e-10 and abs(got[2] - ref[2]) < 1e-10
    assert float(np.max(np.abs(got[0] - ref[0]))) < 1e-10
    assert abs(held - 16 * tiles * 1024) < 12 << 20


# psi held for a few tiles at a time, as grids of more than 2^20 tiles x orbitals have it: parts of one and two
# tiles, and a ragged last part, against the whole and against the same density by P
@pytest.mark.parametrize("functional,ispin", [("PBE", 1), ("PBE", 2), ("TPSS", 1), ("TPSS", 2)])
@pytest.mark.parametrize("nocc", [5, 20])
def test_psi_in_parts(nocc, functional, ispin):
    c = _case(9, 2, functional, ispin, nocc=nocc)
    with lib.Context(c, screen_threshold=0.0) as ctx:
        tiles = ctx.screen_stats()["ntiles"]
        assert tiles > 5
        whole, by_p = ctx.build(), ctx.build_density(c.density_matrix())
        for most in (1, 2, tiles - 1):
            assert lib.lib().pgxc_test_limit_psi(ctx.h, ct.c_int64(most)) == 0
            got = ctx.build()
            for ref, tol in ((whole, 1e-13), (by_p, 1e-11)):
                assert abs(got[1] - ref[1]) < tol * max(1.0, abs(ref[1])) and abs(got[2] - ref[2]) < tol * abs(ref[2])
                assert float(np.max(np.abs(got[0] - ref[0]))) < tol * max(1.0, float(np.max(np.abs(ref[0]))))


@pytest.mark.parametrize("functional,ispin", [("VWN", 1), ("PBE", 1), ("PBE", 2), ("TPSS", 1), ("TPSS", 2)])
def test_gradient_psi_in_parts(functional, ispin):
    c = cases.small_case(functional, seed=49, natoms=9, nrad=9, nang=26, nocc=20, ispin=ispin)
    with lib.Context(c, weighted=False, screen_threshold=0.0) as ctx:
        tiles = ctx.screen_stats()["ntiles"]
        whole = ctx.xc_gradient()
        scale = max(1.0, float(np.max(np.abs(whole[0]))))
        for most in (1, 2, tiles - 1):
            assert lib.lib().pgxc_test_limit_psi(ctx.h, ct.c_int64(most)) == 0
            got = ctx.xc_gradient()
            assert abs(got[1] - whole[1]) < 1e-13 * max(1.0, abs(whole[1]))
            assert float(np.max(np.abs(got[0] - whole[0]))) < 1e-12 * scale


# the gradient on either side of the line between orbitals and P: 5 atoms, 60 functions, so that 16 padded orbitals
# lie below it and 32 and 48 above
@pytest.mark.parametrize("nocc", [4, 30, 40])
@pytest.mark.parametrize("functional,ispin", [("VWN", 1), ("PBE", 1), ("PBE", 2), ("TPSS", 1), ("TPSS", 2)])
def test_gradient_by_orbitals_and_by_p(functional, ispin, nocc):
    c = cases.small_case(functional, seed=50, natoms=5, nrad=12, nang=50, nocc=nocc, ispin=ispin)
    assert c.nbas < 2.3 * 32 and c.nbas > 2.3 * 16
    ref, re = O.xc_gradient(c)
    with lib.Context(c, weighted=False, screen_threshold=0.0) as ctx:
        g, e = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref))))
    assert abs(e - re) < 1e-10 * max(1.0, abs(re))
    np.testing.assert_allclose(g, ref, rtol=0, atol=1e-10 * scale)
