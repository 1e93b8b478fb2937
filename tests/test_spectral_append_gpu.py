"""Page quantizer of the spectral key codec: codes and float32 scales equal, bit for bit, those of the fixed-order sequence
(ascending fused sums, ten refinement rounds with true divisions) written out in numpy."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def _sequence(M, enc, bits, group):
    """M (T, 128) float32, enc (128, 128), bits (128,) -> codes (128, T) int8, scales (128, T / group) float32."""
    acc = np.zeros((M.shape[0], D), np.float32)
    for c in range(D):  # a fused multiply-add rounds once: the float64 product of two float32 numbers is exact
        acc = (acc.astype(np.float64) + M[:, c:c + 1].astype(np.float64) * enc[c][None].astype(np.float64)).astype(np.float32)
    x = np.ascontiguousarray(acc.T).reshape(D, -1, group)
    qmax = np.maximum(2.0 ** (bits.astype(np.float32) - 1) - 1, 1).astype(np.float32)[:, None]
    scale = (np.maximum(np.abs(x).max(-1), np.float32(1e-12)) / qmax).astype(np.float32)

    def code(s):
        return np.minimum(np.maximum(np.rint(x / s[..., None]), -qmax[..., None] - 1), qmax[..., None]).astype(np.float32)

    for _ in range(10):
        q = code(scale)
        num, den = np.zeros_like(scale), np.zeros_like(scale)
        for r in range(group):
            num = num + x[..., r] * q[..., r]
            den = den + q[..., r] * q[..., r]
        scale = np.maximum(num / np.maximum(den, np.float32(1e-12)), np.float32(1e-12)).astype(np.float32)
    used = (bits > 0)[:, None]
    return np.where(used[..., None], code(scale), 0).reshape(D, -1).astype(np.int8), np.where(used, scale, 0).astype(np.float32)


@pytest.mark.parametrize("page,group,dtype,kind,n_used", [
    (128, 64, torch.float16, "normal", 104), (128, 32, torch.bfloat16, "normal", 128), (128, 128, torch.float32, "normal", 17),
    (64, 64, torch.float16, "normal", 96), (64, 8, torch.float32, "normal", 1), (128, 16, torch.float16, "ties", 113),
    (128, 64, torch.float16, "ties", 128), (128, 64, torch.bfloat16, "wide range", 128), (64, 32, torch.float32, "zeros", 64),
    (128, 64, torch.float16, "normal", 0)])
@pytest.mark.parametrize("aligned", [True, False])
def test_codes_and_scales_equal_the_fixed_order_sequence(page, group, dtype, kind, n_used, aligned):
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    rng = np.random.default_rng(page + group + n_used)
    h, n_seq, n_pages = 2, 2, 2
    T = n_pages * page
    enc = np.stack([np.linalg.qr(rng.standard_normal((D, D)))[0] for _ in range(h)]).astype(np.float32)
    M = rng.standard_normal((n_seq, h, T, D)).astype(np.float32) * (np.arange(1, D + 1) ** -0.6).astype(np.float32)
    if kind == "ties":  # directions are channels, values on a coarse grid: quotients fall on halves
        enc = np.stack([np.eye(D, dtype=np.float32)] * h)
        M = rng.integers(-8, 9, M.shape).astype(np.float32) * 0.25
    elif kind == "wide range":
        M = M * np.exp2(rng.integers(-40, 60, (n_seq, h, T, 1))).astype(np.float32)
    elif kind == "zeros":
        M[:, :, : page // 2] = 0
    bits = np.zeros((h, D), np.int64)
    for i in range(h):
        bits[i, rng.permutation(D)[:n_used]] = rng.choice([2, 3, 4, 5, 6, 8], n_used)
    k = torch.from_numpy(M).to(dtype)
    M = k.float().numpy()
    if not aligned:
        wide = torch.zeros(n_seq, h, T, D + 3, dtype=dtype)
        wide[..., 1:1 + D] = k
        k = wide.to(dev)[..., 1:1 + D]
    pack = K.SpectralPackDev(torch.from_numpy(enc), torch.from_numpy(enc), torch.from_numpy(bits), page=page, group=group, device=dev)
    pool = pack.new_pool(n_seq * n_pages)
    slots = torch.arange(n_seq * n_pages, dtype=torch.int32, device=dev)
    K.spectral_append(pack, pool, k.to(dev), slots, n_pages)
    got = K.spectral_dequant_pages(pack, pool, slots, want_k=False)
    codes, scales = got["codes"].cpu().numpy(), got["scales"].cpu().numpy()
    for item in range(n_seq * n_pages):
        s, p = divmod(item, n_pages)
        for i in range(h):
            want_c, want_s = _sequence(M[s, i, p * page:(p + 1) * page], enc[i], bits[i], group)
            assert np.array_equal(codes[item, i], want_c), (item, i, int((codes[item, i] != want_c).sum()))
            assert np.array_equal(scales[item, i].view(np.int32), want_s.view(np.int32)), (item, i)
