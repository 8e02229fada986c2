"""The split backprojector's column-pair staging (planogram rows that are no
multiple of 16 bytes) when every wait on staged data gives up: its four
producer warps leave together, the kernel returns at once, the error word is
set, and the same call afterwards reproduces its result."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["reference", "adjoint"])
def test_pair_staging_gives_up_and_recovers(cuda, mode):
    import torch
    from petl_b200 import Geometry, lib, ops
    L = lib()
    G = Geometry(0.0, 250.0, 48.0, 48.0, 1.5, 0.5, 0.25, volume=(64, 64, 32, 1.5))  # 114 columns
    g = torch.rand(G.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1))
    want = ops.backproject(G, g, mode=mode)
    torch.cuda.synchronize()
    assert L.petl_last_projector_path() == 2 and L.petl_device_error_flag() == 0
    L.petl_force_wait_timeout(1)
    try:
        ops.backproject(G, g, mode=mode)
        torch.cuda.synchronize()
    finally:
        L.petl_force_wait_timeout(0)
    assert L.petl_device_error_flag() == 1
    assert torch.equal(ops.backproject(G, g, mode=mode), want)
    assert L.petl_device_error_flag() == 0


@pytest.mark.parametrize("psi,T", [(0.0, 1.5), (30.0, 1.5), (0.0, 1.6)])
def test_new_planogram_is_zero_where_a_wait_gives_up(cuda, psi, T):
    """A planogram that ops.project allocates holds zeros, not the memory's
    former contents, where the kernels gave up and wrote nothing (the split
    kernels on the axes, for any psi, and for unequal pitch)."""
    import torch
    from petl_b200 import Geometry, lib, ops
    L = lib()
    G = Geometry(psi, 250.0, 48.0, 48.0, T, 0.5, 0.25, volume=(64, 64, 32, 1.5))
    f = torch.rand(G.vol_shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1))
    want = ops.project(G, f)
    torch.cuda.synchronize()
    assert L.petl_device_error_flag() == 0
    old = torch.full(G.shape, float("nan"), device=cuda)  # the allocator hands this block out next
    del old
    L.petl_force_wait_timeout(1)
    try:
        got = ops.project(G, f)
        torch.cuda.synchronize()
    finally:
        L.petl_force_wait_timeout(0)
    assert L.petl_device_error_flag() == 1
    assert torch.isfinite(got).all()
    assert torch.equal(ops.project(G, f), want)
