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
