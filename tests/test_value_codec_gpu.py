"""Hadamard + 2-bit value codes of 16-bit sources (tensor-core transform, thresholds instead of divisions) against the same values
handed over as float32, which take the reference's operation sequence token by token: every byte has to be the same."""

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def _values(kind, n, h, T, dtype, dev):
    g = torch.Generator(device=dev).manual_seed(len(kind))
    v = torch.randn(n, h, T, D, generator=g, device=dev)
    if kind == "sparse":       # few channels: coefficients pile up on few values, many of them near thresholds
        keep = torch.rand(n, h, T, D, generator=g, device=dev) < torch.rand(n, h, T, 1, generator=g, device=dev) * 0.1
        v = torch.where(keep, v, torch.zeros_like(v))
    elif kind == "levels":     # values of one magnitude: exact ties between coefficients
        v = torch.sign(v) * (torch.randint(0, 3, v.shape, generator=g, device=dev) * 0.5)
    elif kind == "extremes":   # zero, tiny, huge, infinite and NaN tokens among ordinary ones
        v[:, :, 0::16] = 0
        v[:, :, 1::16] *= 1e-6
        v[:, :, 2::16] *= 3e-5
        v[:, :, 3::16] *= 5e3 if dtype == torch.float16 else 1e30
        v[:, :, 4::16, 7] = float("inf")
        v[:, :, 5::16, 90] = float("nan")
        v[:, :, 6::16, 1:] = 0
        v[:, :, 7::16] *= 7e3
    return v.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["normal", "sparse", "levels", "extremes"])
def test_codes_equal_the_float32_sequence(kind, dtype):
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    n, h, pages = 3, 5, 11
    v = _values(kind, n, h, pages * 128, dtype, dev)
    signs, cb = K.hadamard_signs(D, 3).to(dev), torch.tensor(K.GAUSSIAN_CODEBOOK[2], device=dev)
    slots = torch.randperm(n * pages, device=dev).to(torch.int32)
    want, got, odd = (K.vblock_pool(h, n * pages, dev) for _ in range(3))
    K.vblock_append(want, v.float(), signs, cb, slots, pages)
    K.vblock_append(got, v, signs, cb, slots, pages)
    # rows that start off the sixteen-byte boundaries (a view into a wider tensor)
    wide = torch.zeros(n, h, pages * 128, D + 5, dtype=dtype, device=dev)
    wide[..., 3:3 + D] = v
    K.vblock_append(odd, wide[..., 3:3 + D], signs, cb, slots, pages)
    assert torch.equal(got, want) and torch.equal(odd, want)
