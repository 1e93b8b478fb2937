"""Page quantizer of layout 1 against the one of layout 0 (the fixed-order sequence with true divisions): the same codes, scales,
coefficients, value indices and norms, bit for bit, for every source type, rank, group, code width and basis shape."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rank,group,kbits,per_head", [(32, 64, 3, True), (32, 32, 4, False), (32, 128, 2, True), (16, 64, 3, False), (16, 128, 4, True),
                                                       (16, 32, 2, True)])
@pytest.mark.parametrize("kind", ["normal", "ties", "extremes"])
def test_both_layouts_hold_the_same_codes(dtype, rank, group, kbits, per_head, kind):
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    n, h, pages = 2, 3, 5
    T = pages * 128
    gen = torch.Generator(device=dev).manual_seed(rank + group + kbits)
    k, v = (torch.randn(n, h, T, 128, generator=gen, device=dev) for _ in range(2))
    basis = torch.randn(h * 128, rank, generator=gen, device=dev) / 16
    if kind == "ties":  # nothing for the low-rank part to take, values on a coarse grid: quotients fall on halves
        k = torch.randint(-7, 8, k.shape, generator=gen, device=dev) * 0.5
        basis[:, 1:] = 0
        basis[:, 0] = 0
    elif kind == "extremes":
        for x in (k, v):
            x[:, :, 3::17] = 0
            x[:, :, 130:200] *= 1e-7
            x[:, :, 260::23] *= 3e3 if dtype == torch.float16 else 1e35
            x[0, 0, 11, 5], x[0, 1, 40, 77], x[1, 2, 70, 127] = float("inf"), float("nan"), float("-inf")
        k[0, 2, :128] = 0
    k, v = k.to(dtype), v.to(dtype)
    signs, cb = K.hadamard_signs(128, 1).to(dev), torch.tensor(K.GAUSSIAN_CODEBOOK[2], device=dev)
    slots = torch.randperm(n * pages, generator=gen, device=dev).to(torch.int32)
    wide = torch.zeros(2, n, h, T, 128 + 3, dtype=dtype, device=dev)
    wide[0, ..., 1:129], wide[1, ..., 1:129] = k, v
    got = []
    for layout, ks, vs in ((0, k, v), (1, k, v), (1, wide[0, ..., 1:129], wide[1, ..., 1:129])):
        g = K.k2b_geom(h, 4, 128, rank, group, h if per_head else 1, kbits, 2, layout)
        pool = K.K2bPool(g, n * pages, dev)
        K.k2b_append(pool, ks, vs, basis, signs, cb, slots, pages)
        got.append(K.k2b_export_stacks(pool, slots))
    for name, want in got[0].items():
        for other in got[1:]:
            same = other[name].view(torch.uint8) == want.view(torch.uint8)
            assert bool(same.all()), f"{name}: {int((~same).sum())} of {same.numel()} bytes differ"
