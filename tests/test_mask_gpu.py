"""The causal-mask test of the prompt attention: one kernel reads a boolean mask once."""

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
