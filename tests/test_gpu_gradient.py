"""Post-SCF XC nuclear gradient on the device (pgxc_xc_gradient) against the
oracle's independent restatement (itself checked against finite differences
in tests/test_gradient.py); every layout, both spins, LDA, GGA and meta-GGA."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from pgxc import cases, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [("fp64", -1.0), ("fp64", 0.0), ("mixed", 1e-10)],
                         ids=["dense", "screened", "int8-screened"])
@pytest.mark.parametrize("xc,ispin,lmax", [("VWN", 1, 2), ("PBE", 1, 3), ("BLYP", 1, 2), ("PBE", 2, 2),
                                           ("B3LYP", 2, 3), ("HCTH407", 1, 2)])
def test_gradient_matches_oracle(xc, ispin, lmax, layout):
    precision, thr = layout
    if ispin == 2 and thr < 0:
        pytest.skip("the dense layout is closed shell")
    case = cases.small_case(functional=xc, seed=62, natoms=4, nocc=5, ispin=ispin, lmax=lmax)
    ref, re = O.xc_gradient(case)
    with lib.Context(case, weighted=False, precision=precision, screen_threshold=thr) as ctx:
        g, e = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref))))
    assert abs(e - re) < 1e-10 * max(1.0, abs(re))
    np.testing.assert_allclose(g, ref, rtol=0, atol=1e-10 * scale)
    np.testing.assert_allclose(g.sum(0), 0.0, atol=1e-9 * scale)


@pytest.mark.parametrize("layout", [("fp64", 0.0), ("mixed", 1e-10)], ids=["screened", "int8-screened"])
@pytest.mark.parametrize("xc,ispin", [("TPSS", 1), ("TPSS", 2), ("M06L", 2), ("VSXC", 1)])
def test_mgga_gradient_matches_oracle(xc, ispin, layout):
    """Meta-GGAs: tau and df/dtau per point, and the tau terms (d_k d_j phi Y_j)
    in the orbital sums; the oracle's form is checked against finite
    differences in tests/test_gradient.py."""
    precision, thr = layout
    case = cases.small_case(functional=xc, seed=64, natoms=4, nocc=5, ispin=ispin, lmax=2)
    ref, re = O.xc_gradient(case)
    with lib.Context(case, weighted=False, precision=precision, screen_threshold=thr) as ctx:
        g, e = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref))))
    assert abs(e - re) < 1e-10 * max(1.0, abs(re))
    np.testing.assert_allclose(g, ref, rtol=0, atol=1e-10 * scale)
    np.testing.assert_allclose(g.sum(0), 0.0, atol=1e-9 * scale)


@pytest.mark.parametrize("xc,ispin", [("VWN", 1), ("PBE", 2), ("TPSS", 1)])
def test_core_terms_do_not_round_the_gradient(xc, ispin):
    """What a function contributes on its own atom's points leaves and enters the
    same atom.  With core functions (exponents up to 1e4) those terms are the
    largest by far; a gradient that does not carry them has a sum over atoms,
    and a difference between two calls, of the rounding of the other terms
    alone: tiles (300) x eps (1.1e-16) of the largest component, three times over."""
    case = cases.build_case("core", ["C", "H", "O", "H"], np.array([[0, 0, 0], [2.1, 0, 0], [0, 2.3, 0], [0, 0, 2.0]]),
                            seed=5, exp_range=(0.05, 1e4), nrad=50, nang=194, functional=xc, nocc=8, ispin=ispin,
                            orthonormalise=False)
    with lib.Context(case, weighted=False) as ctx:
        a, b = ctx.xc_gradient()[0], ctx.xc_gradient()[0]
    scale = float(np.max(np.abs(a)))
    assert float(np.max(np.abs(a.sum(0)))) < 1e-13 * scale
    assert float(np.max(np.abs(a - b))) < 1e-13 * scale


def test_gradient_of_many_chunks():
    """200 atoms with f shells, about 70 chunks of slot rows: the lists are made chunk by
    chunk, so what the context holds after a gradient is one chunk's rows (at most
    4 GB), the weight term's scratch (at most 2 GB) and arrays by point, not the
    lists of the whole grid (0.4 GB here).  Two halves of the grid, chunked in
    their own way, sum to the whole; a second call finds the chunks again."""
    import torch
    n = 200
    rng = np.random.default_rng(21)
    els, xyz = cases.random_cluster(rng, [("C", 80), ("H", 60), ("O", 40), ("N", 20)], 18.0, 1.0)
    case = cases.build_case("many", els, xyz, seed=21, exp_range=(0.05, 1e4), nrad=50, nang=194, functional="VWN",
                            nocc=16, shells=cases.SHELLS_F, orthonormalise=False)
    torch.cuda.init()
    with lib.Context(case, weighted=False, screen_threshold=1e-10) as ctx:
        free = torch.cuda.mem_get_info()[0]
        g, e = ctx.xc_gradient()
        held = free - torch.cuda.mem_get_info()[0]
        again, _ = ctx.xc_gradient()
    points = (case.npts + 127) // 128 * 128
    weights = points
    while 28 * n * weights > 2e9:
        weights = (weights // 2 + 127) // 128 * 128
    assert held < 4.0e9 + 28 * n * weights + 0.35e9
    scale = float(np.max(np.abs(g)))
    assert float(np.max(np.abs(again - g))) < 1e-12 * scale
    half = np.zeros_like(g)
    for pick in (slice(0, case.npts // 2), slice(case.npts // 2, None)):
        c = dataclasses.replace(case, grid_xyz=case.grid_xyz[pick], grid_wraw=case.grid_wraw[pick],
                                point_atom=case.point_atom[pick])
        with lib.Context(c, weighted=False, screen_threshold=1e-10) as ctx:
            gh, eh = ctx.xc_gradient()
        half += gh
        e -= eh
    assert abs(e) < 1e-10
    assert float(np.max(np.abs(half - g))) < 1e-11 * scale


@pytest.mark.parametrize("layout", [("fp64", -1.0), ("fp64", 0.0), ("mixed", 1e-10)],
                         ids=["dense", "screened", "int8-screened"])
def test_first_gradient_allocates_twice(layout):
    """A gradient is asked for once per geometry, so the first call counts: the
    tables of its lists (by tile, small) and its scratch are all that it
    allocates, and nothing is released (each large allocation takes 0.35 ms)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    precision, thr = layout
    case = cases.small_case(functional="PBE", seed=65, natoms=6, nrad=50, nang=194)
    with lib.Context(case, weighted=False, precision=precision, screen_threshold=thr) as ctx:
        ctx.build()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
            ctx.xc_gradient()
        names = [e.name for e in prof.events()]
    if "cudaLaunchKernel" not in names:
        pytest.skip("the profiler records no runtime calls here")
    assert names.count("cudaMalloc") <= 2 and "cudaFree" not in names


def test_gradient_without_room_for_psi():
    """No room for psi beside the rows: the gradient takes P, and a second one does not ask again."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    case = cases.small_case(functional="PBE", seed=68, natoms=12, nrad=160, nang=194, nocc=40)
    torch.cuda.init()
    with lib.Context(case, weighted=False, screen_threshold=0.0) as ctx:
        tiles = ctx.screen_stats()["ntiles"]
        assert 48 * tiles * 1024 > 112 << 20
        many, case.nocc = case.nocc, 1
        ctx.xc_gradient(C=case.C[:, :1, 0].T, occ=case.occ[:1, 0])  # the scratch, with psi of 16 orbitals
        case.nocc = many
        torch.cuda.empty_cache()
        taken = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
        got = ctx.xc_gradient()
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
            again = ctx.xc_gradient()
        names = [e.name for e in prof.events()]
        del taken
        torch.cuda.empty_cache()
    with lib.Context(case, weighted=False, screen_threshold=0.0) as ctx:
        ref = ctx.xc_gradient()
    scale = max(1.0, float(np.max(np.abs(ref[0]))))
    for g, e in (got, again):
        assert abs(e - ref[1]) < 1e-11 * max(1.0, abs(ref[1]))
        np.testing.assert_allclose(g, ref[0], rtol=0, atol=1e-11 * scale)
    assert "cudaMalloc" not in names and "cudaFree" not in names


@pytest.mark.parametrize("npts", [129, (1 << 17) - 1, 1 << 17])
def test_dense_gradient_in_either_point_order(npts):
    """The dense layout's gradient takes the points as they lie up to 2^17 of them
    and in Morton order from there on; the last tile is ragged.  Against the
    screened context, whose points are always in Morton order."""
    case = cases.small_case(functional="PBE", seed=67, natoms=4, nrad=250, nang=194, nocc=5)
    assert case.npts >= npts
    pick = np.sort(np.random.default_rng(9).permutation(case.npts)[:npts])
    case = dataclasses.replace(case, grid_xyz=case.grid_xyz[pick], grid_wraw=case.grid_wraw[pick],
                               point_atom=case.point_atom[pick])
    r = []
    for thr in (-1.0, 0.0):
        with lib.Context(case, weighted=False, screen_threshold=thr) as ctx:
            r.append(ctx.xc_gradient())
    scale = max(1.0, float(np.max(np.abs(r[1][0]))))
    assert abs(r[0][1] - r[1][1]) < 1e-11 * max(1.0, abs(r[1][1]))
    np.testing.assert_allclose(r[0][0], r[1][0], rtol=0, atol=1e-11 * scale)


def test_gradient_needs_the_raw_grid():
    case = cases.small_case(functional="PBE", seed=63)
    O.weight_case(case)
    with lib.Context(case, screen_threshold=0.0) as ctx:
        with pytest.raises(lib.PgxcError):
            ctx.xc_gradient()
