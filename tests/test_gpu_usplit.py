"""The split forward for unequal voxel height and u1 pitch on an axis-aligned
planogram against the FP64 oracle and the general kernels: bins taller and
lower than voxels (0 to 3 whole voxels in a bin, the unrolled forms, and
more), calls too small for the split form (a ray per thread), psi = 0 and 90,
ragged and off-centre volumes, rays that miss the volume on most planes, a
volume wider than the panels, view subsets, slope ranges and the MLEM ratio."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2
from helpers import ellipsoids

pytestmark = pytest.mark.gpu

CASES = {
    # psi, D, L, H, T, v_m0, v_m1 ; volume (x, y, z, width, height, offsets) ; path (3 split, 0 general)
    "petx0": ((0.0, 101.0, 120.0, 60.0, 1.6, 0.99, 0.55), (40, 36, 30, 0.5, 0.5), 3),
    "petx90": ((90.0, 120.0, 80.0, 60.0, 1.6, 0.7, 0.45), (36, 41, 33, 0.5, 0.5, 2.0, -1.0, 3.0), 3),
    "low_bins": ((0.0, 100.0, 50.0, 30.0, 1.0, 0.5, 0.25), (30, 40, 12, 2.0, 2.7), 3),
    "one_whole": ((90.0, 100.0, 75.0, 27.0, 1.5, 0.45, 0.2), (52, 60, 18, 1.5, 1.1, 3.0, -4.5, 1.5), 3),
    "two_whole": ((0.0, 100.0, 40.0, 44.0, 2.0, 0.4, 0.2), (50, 20, 61, 0.9, 0.75), 3),
    "four_whole": ((0.0, 100.0, 40.0, 44.0, 2.0, 0.4, 0.2), (30, 20, 90, 1.0, 0.45), 3),
    "few_rays": ((0.0, 40.0, 12.0, 10.0, 1.6, 0.5, 0.25), (14, 12, 9, 1.0, 1.2, 1.0, 0.0, -2.0), 3),
    "few_rays90": ((90.0, 40.0, 12.0, 10.0, 1.6, 0.5, 0.25), (13, 15, 21, 0.6, 0.45, -1.0, 2.0, 0.0), 3),
    "too_many_rows": ((0.0, 100.0, 40.0, 44.0, 4.0, 0.4, 0.2), (30, 20, 90, 1.0, 0.45), 0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_unequal_pitch_forward(cuda, name):
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol, path = CASES[name]
    G, Go = Geometry(*args, volume=vol), O.make_geom(*args, vol)
    rng = np.random.default_rng(2)
    f = ellipsoids(G.vol_shape, (vol[3], vol[4]), rng, 6) + 0.1 * rng.random(G.vol_shape).astype(np.float32)
    ft = torch.from_numpy(f).to(cuda)
    a = ops.project(G, ft)
    assert lib().petl_last_projector_path() == path
    assert rel_l2(a.cpu().numpy(), O.project(Go, f)[0]) < 1e-5
    meas = torch.rand(G.shape, device=cuda)
    sub, v1 = (1, 3), (2, G.shape[0] - 1)
    out = []
    for d in (0, 1):
        try:
            lib().petl_set_dispatch(d)
            out.append([ops.project(G, ft, torch.full(G.shape, -7.0, device=cuda), subset=sub, v1_range=v1),
                        ops.project_ratio(G, ft, meas, torch.full(G.shape, -7.0, device=cuda), subset=sub, v1_range=v1)])
        finally:
            lib().petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert lib().petl_device_error_flag() == 0
    for x, y in zip(*out):
        assert torch.equal(x == -7.0, y == -7.0)
    assert torch.equal(out[0][0] == 0, out[1][0] == 0)  # rays that meet no voxel stay exactly zero
    assert rel_l2(out[0][0].cpu().numpy(), out[1][0].cpu().numpy()) < 1e-5
    # the ratio where the ray meets more than the rim of a voxel
    ok = out[1][0] > 0.05 * out[1][0].max()
    assert rel_l2(out[0][1][ok].cpu().numpy(), out[1][1][ok].cpu().numpy()) < 1e-5


@pytest.mark.parametrize("name", list(CASES))
def test_unequal_pitch_adjoint_has_the_forward_weights(cuda, name):
    """Single weights of P and of P^T: the column P e_j of a voxel against the
    rows P^T e_i of bins along it.  Either side rounds a weight a handful of
    times (its u0 and u1 part and three factors): 4e-7 of the largest weight.
    Weights from positions in float differ by up to 1e-5 here."""
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol, path = CASES[name]
    G = Geometry(*args, volume=vol)
    gen = torch.Generator().manual_seed(4)
    nz, ny, nx = G.vol_shape
    worst = 0.0
    for k in range(4):
        # corners and the middle of the volume
        j = ((nz // 2, ny // 2, nx // 2), (1, 2, nx - 2), (nz - 2, ny - 1, 3), (nz // 3, 0, nx // 2))[k]
        f = torch.zeros(G.vol_shape, device=cuda)
        f[j] = 1.0
        col = ops.project(G, f)
        bins = torch.nonzero(col.reshape(-1) > 0.02 * col.max()).reshape(-1).cpu()
        if len(bins) == 0:
            continue
        for i in bins[torch.randint(len(bins), (8,), generator=gen)].tolist():
            g = torch.zeros(G.shape, device=cuda)
            g.view(-1)[i] = 1.0
            row = ops.backproject(G, g, mode="adjoint")
            worst = max(worst, abs(float(row[j]) - float(col.view(-1)[i])) / float(col.max()))
    assert lib().petl_device_error_flag() == 0
    assert worst < 4e-7, worst


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("sub,v1", [(None, None), ((1, 3), (2, -1))])
def test_unequal_pitch_adjoint_against_oracle(cuda, name, sub, v1):
    """Voxels of P^T g, with accumulation and scale, against 64 bits: voxel j is
    <P e_j, g>, with P e_j from the oracle."""
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol, path = CASES[name]
    G, Go = Geometry(*args, volume=vol), O.make_geom(*args, vol)
    rng = np.random.default_rng(6)
    g = rng.random(G.shape).astype(np.float32)
    r1 = None if v1 is None else (v1[0], G.shape[0] + v1[1])
    keep = np.zeros(G.shape, bool)
    keep[slice(*r1) if r1 else slice(None), slice(sub[0], None, sub[1]) if sub else slice(None)] = True
    gk = np.where(keep, g, 0.0).astype(np.float64)
    f0 = torch.ones(G.vol_shape, device=cuda)
    got = ops.backproject(G, torch.from_numpy(g).to(cuda), f0, mode="adjoint", subset=sub, v1_range=r1,
                          accumulate=True, scale=0.5).cpu().numpy()
    assert lib().petl_last_projector_path() == 0 and lib().petl_device_error_flag() == 0
    nz, ny, nx = G.vol_shape
    for j in ((nz // 2, ny // 2, nx // 2), (0, 0, 0), (nz - 1, ny - 1, nx - 1), (1, ny // 3, nx - 2), (nz - 2, 1, 2)):
        e = np.zeros(G.vol_shape, np.float32)
        e[j] = 1.0
        want = 1.0 + 0.5 * float((np.asarray(O.project(Go, e)[0], np.float64) * gk).sum())
        assert abs(float(got[j]) - want) < 1e-5 * want, (j, got[j], want)
