"""Contiguous tensors that start at an odd element of their allocation: the
projectors of every kernel family give what they give for aligned ones (bit
for bit where the same kernels run; where a staged copy needs an aligned
base, another family's sums in another order), or refuse them."""
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "axis": ((0.0, 128.0, 64.0, 32.0, 2.0, 0.5, 0.25), (32, 36, 16, 2.0)),
    "axis90": ((90.0, 128.0, 64.0, 32.0, 2.0, 0.5, 0.25), (36, 32, 16, 2.0)),
    "steep": ((0.0, 60.0, 48.0, 60.0, 1.5, 0.5, 0.7), (32, 48, 24, 1.5)),
    "rotated": ((30.0, 128.0, 64.0, 32.0, 2.0, 0.5, 0.25), (32, 36, 16, 2.0)),
    "pitch": ((0.0, 128.0, 64.0, 32.0, 2.0, 0.5, 0.25), (32, 36, 16, 1.5, 1.25)),
}


def _off(x, k=1):
    import torch
    b = torch.zeros(x.numel() + k, device=x.device, dtype=x.dtype)
    v = b[k:].view(x.shape)
    v.copy_(x)
    assert v.data_ptr() % (2 * x.element_size()) != 0 and v.is_contiguous()
    return v


@pytest.mark.parametrize("dispatch", [0, 1, 2, 3])
@pytest.mark.parametrize("name", list(CASES))
def test_projectors_on_offset_views(cuda, name, dispatch):
    import torch
    from petl_b200 import Geometry, lib, ops
    args, vol = CASES[name]
    G = Geometry(*args, volume=vol)
    gen = torch.Generator(device=cuda).manual_seed(3)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen)
    g = torch.rand(G.shape, device=cuda, generator=gen)
    try:
        assert lib().petl_set_dispatch(dispatch) == 0
        a = [ops.project(G, f), ops.project_ratio(G, f, g, torch.zeros_like(g)), ops.backproject(G, g),
             ops.backproject(G, g, mode="adjoint")]
        b = [ops.project(G, _off(f), _off(torch.zeros_like(g))),
             ops.project_ratio(G, _off(f), _off(g), _off(torch.zeros_like(g))), ops.backproject(G, _off(g), _off(f)),
             ops.backproject(G, _off(g), _off(f), mode="adjoint")]
        # one of the ratio's two planograms alone
        c = [ops.project_ratio(G, f, _off(g), torch.zeros_like(g)), ops.project_ratio(G, f, g, _off(torch.zeros_like(g)))]
    finally:
        lib().petl_set_dispatch(0)
    torch.cuda.synchronize()
    assert lib().petl_device_error_flag() == 0
    for x, y in zip(a, b):
        assert float((x - y).norm() / x.norm()) < 1e-6
    if dispatch == 0:  # the forward stages its own copy of the volume: the same kernels run
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    assert torch.equal(a[1], c[0]) and torch.equal(a[1], c[1])


def test_bf16_projector_on_offset_views(cuda):
    import torch
    from petl_b200 import Geometry, PetlError, ops
    args, vol = CASES["axis"]
    G = Geometry(*args, volume=vol)
    gen = torch.Generator(device=cuda).manual_seed(3)
    f = torch.rand(G.vol_shape, device=cuda, generator=gen).bfloat16()
    g = torch.rand(G.shape, device=cuda, generator=gen).bfloat16()
    want = ops.project_bf16(G, f)
    assert torch.equal(ops.project_bf16(G, _off(f), _off(torch.zeros_like(g))), want)
    assert torch.equal(ops.project_ratio_bf16(G, f, _off(g), _off(torch.zeros_like(g))), ops.project_ratio_bf16(G, f, g))
    with pytest.raises(PetlError):
        ops.backproject_bf16(G, _off(g))
