"""The causal-mask test of the prompt attention (one kernel reads a boolean mask once), and what the attention does with the mask."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_q,S", [(1, 1), (7, 7), (5, 133), (64, 2048), (33, 4111), (300, 300)])
def test_only_the_plain_causal_mask_passes(n_q, S):
    from bmx_b200.packed_streaming import PackedStreamingLayer

    dev = torch.device("cuda:0")
    is_causal = PackedStreamingLayer._mask_is_causal
    base = torch.ones(n_q, S, dtype=torch.bool, device=dev).tril(S - n_q)
    wide = torch.zeros(2, 1, n_q, S + 5, dtype=torch.bool, device=dev)
    wide[..., 3:3 + S] = base
    for m in (base[None, None], base[None, None].expand(3, 1, n_q, S), base[None, None].repeat(2, 1, 1, 1), wide[..., 3:3 + S]):
        assert is_causal(m, n_q, S)
        for b, i, j in ((0, 0, 0), (m.shape[0] - 1, n_q - 1, S - 1), (0, n_q // 2, S // 2), (m.shape[0] - 1, 0, S - 1)):
            other = m.clone()
            other[b, 0, i, j] ^= True
            assert not is_causal(other, n_q, S), (b, i, j)
    assert not is_causal(base[None, None][..., : S - 1], n_q, S)


@pytest.mark.parametrize("n_q,S", [(3, 64), (3, 61), (40, 4096)])
def test_any_byte_but_zero_is_true(n_q, S):
    """The answer does not depend on which byte stands for true, in the wide loop (rows on 16-byte boundaries) as in the other."""
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    ones = torch.ones(n_q, S, dtype=torch.uint8, device=dev).tril(S - n_q)[None, None]
    for byte in (1, 2, 0x80, 0xFF):
        mask = ones * byte
        assert K.mask_is_causal(mask.view(torch.bool), n_q, S), byte
        mask[0, 0, 0, 1] = 0
        assert not K.mask_is_causal(mask.view(torch.bool), n_q, S), byte
        mask[0, 0, 0, 1] = byte
        mask[0, 0, 0, S - 1] = byte
        assert not K.mask_is_causal(mask.view(torch.bool), n_q, S), byte


@pytest.mark.parametrize("n_q", [1, 5, 70])
def test_a_causal_mask_may_be_anywhere_and_laid_out_anyhow(n_q):
    """The plain causal mask on the host, as a transposed view, as a slice of a wider one or expanded over the sequences gives the
    same attention as one on the device in one piece."""
    from types import SimpleNamespace

    from bmx_b200.packed_streaming import PackedStreamingLayer
    from bmx_b200.recipes import spec_pair

    dev = torch.device("cuda:0")
    B, h, G, S = 2, 2, 2, 400 + n_q
    config = SimpleNamespace(num_attention_heads=h * G, num_key_value_heads=h, head_dim=128, hidden_size=h * G * 128, max_position_embeddings=4096,
                             rope_theta=5e5, rope_parameters={"rope_type": "default", "rope_theta": 5e5}, standardize_rope_params=lambda: None)
    gen = torch.Generator(device=dev).manual_seed(n_q)
    layer = PackedStreamingLayer(*spec_pair("kivi", group=64), config, recent_window=64)
    k, v = (torch.randn(B, h, S, 128, generator=gen, device=dev).half() for _ in range(2))
    layer.update(k, v)
    q = torch.randn(B, h * G, n_q, 128, generator=gen, device=dev).half()
    base = torch.ones(n_q, S, dtype=torch.bool, device=dev).tril(S - n_q)[None, None]
    wide = torch.zeros(1, 1, n_q, S + 5, dtype=torch.bool, device=dev)
    wide[..., 3:3 + S] = base
    want = layer.attend(q, 128 ** -0.5, is_causal=True, attention_mask=base)
    assert bool(want.isfinite().all())
    masks = {"host": base.cpu(), "host, both": base.cpu().expand(B, 1, n_q, S), "both": base.expand(B, 1, n_q, S), "slice": wide[..., 3:3 + S],
             "transposed": base.transpose(2, 3).contiguous().transpose(2, 3)}
    for name, mask in masks.items():
        assert torch.equal(layer.attend(q, 128 ** -0.5, is_causal=True, attention_mask=mask), want), name
