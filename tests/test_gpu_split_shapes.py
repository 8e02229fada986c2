"""The split z kernels' launch shapes against the single-pass and
first-generation shear kernels (dispatch 3), which do the same float
operations in the same order: bit equality is the bound.  The launch counts
show that the split kernels ran (an x pass beside the z pass, and a record
kernel in the backward, that the others do not have); which launch shape each
case takes is in tests/test_split_bounds.py.  The cases sit where
a shape or a rule changes: slopes steeper than one row per plane or slope
(two per warp), planogram rows that are no multiple of 16 bytes (staged by
column pairs), few tiles (four consumer warps, one or two CTAs per SM), slope tails of one group,
half a block and more, ragged and off-centre volumes, masked columns on
either side, psi = 90, view subsets and slope ranges."""
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # psi, D, L, H, T, v_m0, v_m1 ; volume
    "tail1_u0mod2": ((0.0, 250.0, 48.0, 48.0, 1.5, 0.5, 0.25), (64, 64, 32, 1.5)),          # (33, 83, 32, 114)
    "steep_slopes": ((0.0, 100.0, 72.0, 72.0, 1.5, 0.5, 0.25), (96, 96, 48, 1.5)),          # 1.4 rows per slope
    "steep_planes": ((0.0, 60.0, 60.0, 90.0, 2.0, 0.6, 1.0), (40, 36, 45, 2.0)),            # 0.93 rows per plane
    "steeper_planes": ((0.0, 60.0, 60.0, 120.0, 2.0, 0.6, 1.6), (40, 60, 100, 2.0)),        # 1.6 rows per plane
    "steepest_planes": ((0.0, 60.0, 64.0, 190.0, 2.0, 0.6, 2.5), (36, 58, 98, 2.0)),         # 2.5, 50-column rows
    "tall_voxels": ((0.0, 120.0, 60.0, 60.0, 2.0, 0.6, 0.5), (60, 130, 30, 2.0)),           # steep, 66-column rows
    "rag90": ((90.0, 115.0, 71.0, 65.0, 1.5, 0.45, 0.2), (75, 71, 38, 1.5, 1.5, 3.0, -4.5, 1.5)),
    "few_tiles": ((0.0, 250.0, 48.0, 56.0, 1.5, 0.5, 0.25), (64, 64, 32, 1.5)),             # a subset of 8: two CTAs per SM
    "wide": ((0.0, 300.0, 128.0, 32.0, 1.0, 0.5, 0.25), (130, 40, 20, 1.0)),                # 278 columns, volume narrower
    "one_row_block": ((0.0, 128.0, 64.0, 13.0, 1.0, 0.3, 0.1), (30, 34, 11, 1.0, 1.0, 6.0, 0.0, 0.0)),
}


@pytest.mark.parametrize("sub,v1", [(None, None), ((1, 3), None), ((2, 8), (1, -2))])
@pytest.mark.parametrize("name", list(CASES))
def test_split_shapes_equal_single_pass(cuda, name, sub, v1):
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol = CASES[name]
    G = Geometry(*args, volume=vol)
    gen = torch.Generator(device=cuda).manual_seed(7)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen)
    g = torch.rand(G.shape, device=cuda, generator=gen)
    rng = None if v1 is None else (v1[0], G.shape[0] + v1[1])
    out, launches = {}, {}
    L = lib()

    def counted(d, fn):
        n = L.petl_launch_count()
        out[d].append(fn())
        launches[d].append(L.petl_launch_count() - n)

    try:
        for d in (0, 3):
            assert L.petl_set_dispatch(d) == 0
            out[d], launches[d] = [], []
            counted(d, lambda: ops.project(G, f, torch.full(G.shape, 7.0, device=cuda), subset=sub, v1_range=rng))
            counted(d, lambda: ops.project_ratio(G, f, g, torch.full(G.shape, 7.0, device=cuda), subset=sub, v1_range=rng))
            for m in ("reference", "adjoint"):
                counted(d, lambda: ops.backproject(G, g, subset=sub, v1_range=rng, mode=m))
    finally:
        L.petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert L.petl_device_error_flag() == 0
    assert [a - b for a, b in zip(launches[0], launches[3])] == [1, 1, 2, 2]  # the split kernels ran
    for i, (a, b) in enumerate(zip(out[0], out[3])):
        if "planes" in name and i >= 2:  # dispatch 3 takes the first-generation backprojector: another order
            assert float((a - b).norm() / b.norm()) < 1e-6
        else:
            assert torch.equal(a, b), i


@pytest.mark.parametrize("nx,nz,acc", [(64, 32, False), (61, 33, True), (50, 70, False), (132, 70, True), (131, 65, False)])
def test_flat_backprojection_shapes(cuda, nx, nz, acc):
    """One slope at v1 = 0: ragged x (blocks of 2 and of 8), z (pairs and
    blocks of 32 and of 64), accumulation, both modes, volumes on either side of
    the rule for small ones; bit equality with the single-pass kernel."""
    import torch
    from petl_b200 import Geometry, lib, ops
    G = Geometry(0.0, 128.0, 64.0, 1.5 * nz, 1.5, 0.5, 0.25, volume=(nx, 57, nz, 1.5, 1.5, 3.0, 0.0, 0.0)).rebinned()
    gen = torch.Generator(device=cuda).manual_seed(3)
    g = torch.rand(G.shape, device=cuda, generator=gen)
    f0 = torch.rand(G.vol_shape, device=cuda, generator=gen)
    out, launches = {}, {}
    try:
        for d in (0, 3):
            lib().petl_set_dispatch(d)
            n = lib().petl_launch_count()
            out[d] = [ops.backproject(G, g, f0.clone(), mode=m, accumulate=acc, scale=0.7) for m in ("reference", "adjoint")]
            launches[d] = lib().petl_launch_count() - n
    finally:
        lib().petl_set_dispatch(0)
    assert launches[0] == launches[3] + 2  # z sums and gather in each
    for a, b in zip(out[0], out[3]):
        assert torch.equal(a, b)


# Shift steps a rounding error below one row: the exact steps differ by less
# than a row, the tabulated shifts (v1 and y are floats) by two in places.
NEAR_ONE_ROW = {
    # slopes 8..11 on plane 0: -116, -116, -115, -113
    "slopes": ((0.0, 214.36044311523438, 18.4, 180.48056, 0.92, 0.02, 0.7152043),
               (24, 234, 114, 0.92, 0.92, 0.0, 0.0, 0.00013313642136), None),
    # planes 20..23 of slope 0: -296, -295, -295, -293
    "planes": ((0.0, 167.48048400878906, 15.8, 385.2051086425781, 0.79, 0.02, 1.0),
               (24, 208, 60, 0.79, 0.79, 0.0, 0.0, -0.3948222875649961), (0, 64)),
}


@pytest.mark.parametrize("name", list(NEAR_ONE_ROW))
def test_shift_steps_near_one_row(cuda, name):
    """Every plane and slope counts where neighbouring shifts differ by two
    rows although their step is below one: bit equality with dispatch 3 for
    the forward; the backward there takes the first-generation kernel, whose
    sums of at most 64 x 5 terms in another order differ by rounding."""
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol, rng = NEAR_ONE_ROW[name]
    G = Geometry(*args, volume=vol)
    gen = torch.Generator(device=cuda).manual_seed(11)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen)
    g = torch.rand(G.shape, device=cuda, generator=gen)
    L = lib()
    out = {}
    try:
        for d in (0, 3):
            assert L.petl_set_dispatch(d) == 0
            n = L.petl_launch_count()
            x = ops.project(G, f, torch.zeros(G.shape, device=cuda), v1_range=rng)
            n1 = L.petl_launch_count()
            out[d] = (n1 - n, x, [ops.backproject(G, g, v1_range=rng, mode=m) for m in ("reference", "adjoint")])
    finally:
        L.petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert L.petl_device_error_flag() == 0
    assert out[0][0] == out[3][0] + 1  # the split forward ran: two passes
    assert torch.equal(out[0][1], out[3][1])
    for a, b in zip(out[0][2], out[3][2]):
        assert float((a - b).norm() / b.norm()) < 1e-6


@pytest.mark.parametrize("slopes", [72, 74])
@pytest.mark.parametrize("rows", [250, 320])
def test_steep_slopes_on_tall_panels(cuda, slopes, rows):
    """1.2 rows per slope on planograms of more than 240 rows, without a tail
    of slopes (72) and with one of a single group (74): the split forward
    takes both, equal to the single-pass or first-generation form."""
    import torch
    from petl_b200 import Geometry, lib, ops
    # R = 24.6 bins, volume of 60 planes: step = 29.5 / 24.6
    G = Geometry(0.0, 49.2, 20.0, float(rows), 1.0, 0.2, 1.52, volume=(24, 60, 40, 1.0))
    assert G.shape[0] >= slopes and G.shape[2] == rows
    gen = torch.Generator(device=cuda).manual_seed(5)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen)
    L = lib()
    out, launches = {}, {}
    try:
        for d in (0, 3):
            assert L.petl_set_dispatch(d) == 0
            n = L.petl_launch_count()
            out[d] = ops.project(G, f, torch.full(G.shape, 7.0, device=cuda), v1_range=(0, slopes))
            launches[d] = L.petl_launch_count() - n
    finally:
        L.petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert L.petl_device_error_flag() == 0
    assert launches[0] == launches[3] + 1  # the split forward ran: two passes
    assert torch.equal(out[0], out[3])


def test_more_rows_than_fifteen_thousand(cuda):
    """Long thin volumes and panels keep the split kernels (row indexes are
    plain integers throughout)."""
    import torch
    from petl_b200 import Geometry, lib, ops
    rows = 16400
    G = Geometry(0.0, 40.0, 4.0, float(rows), 1.0, 0.1, 0.26, volume=(8, 10, rows, 1.0))
    assert G.shape[2] == rows and G.shape[0] >= 10
    gen = torch.Generator(device=cuda).manual_seed(9)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen)
    g = torch.rand(G.shape, device=cuda, generator=gen)
    L = lib()
    out = {}
    try:
        for d in (0, 3):
            assert L.petl_set_dispatch(d) == 0
            n = [L.petl_launch_count()]
            x = ops.project(G, f)
            n.append(L.petl_launch_count())
            y = ops.backproject(G, g)
            n.append(L.petl_launch_count())
            out[d] = (x, y, n[1] - n[0], n[2] - n[1])
    finally:
        L.petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert L.petl_device_error_flag() == 0
    assert out[0][2] == out[3][2] + 1 and out[0][3] == out[3][3] + 2  # the split kernels ran
    assert torch.equal(out[0][0], out[3][0])
    assert float((out[0][1] - out[3][1]).norm() / out[3][1].norm()) < 1e-6
