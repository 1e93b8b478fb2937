"""GPU parity of the plain-RTN path (bmx arms rtn_token / rtn_channel): every codec stage is
elementwise, so codes and fp16 scales must equal the oracle's bit for bit; attention within 2e-3."""

import math

import numpy as np
import pytest
import torch

from oracle import bmx_oracle as O
from tests.helpers import golden

pytestmark = pytest.mark.gpu
D = 128


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch.device("cuda:0")


def _inputs(seed, n_seq, h_kv, T):
    g = torch.Generator().manual_seed(seed)
    k = torch.randn(n_seq, h_kv, T, D, generator=g)
    k[..., :4] *= 8.0  # outlier channels, as in the RTN benchmark configuration
    return k.half().contiguous(), torch.randn(n_seq, h_kv, T, D, generator=g).half().contiguous()


def _oracle_blocks(k, v, s, p, page, k_arm, kg, vg, kbits):
    Mk = O.to_matrix(k[s, :, p * page:(p + 1) * page].float().numpy())
    Mv = O.to_matrix(v[s, :, p * page:(p + 1) * page].float().numpy())
    kp, _ = O.quantize_packed(k_arm, Mk, bits=kbits, group=kg)
    vp, _ = O.quantize_packed("rtn_token", Mv, bits=2, group=vg)
    return kp, vp


@pytest.mark.parametrize("page,k_arm,kg,vg,kbits", [(128, "rtn_channel", 32, 32, 4), (128, "rtn_token", 32, 32, 4),
                                                     (64, "rtn_channel", 64, 64, 2), (64, "rtn_token", 64, 128, 3),
                                                     (128, "rtn_token", 128, 32, 4)])
def test_append_codes_and_scales_bit_exact(page, k_arm, kg, vg, kbits):
    from bmx_b200 import kernels as K
    dev = _dev()
    h_kv, n_seq, n_pg = 2, 2, 2
    k, v = _inputs(3, n_seq, h_kv, n_pg * page)
    g = K.rtn_geom(h_kv, 4, page, k_arm, kg, vg, kbits, 2)
    pool = K.RtnPool(g, 8, dev)
    slots = torch.tensor([6, 1, 3, 4], dtype=torch.int32, device=dev)
    K.rtn_append(pool, k.to(dev), v.to(dev), slots, n_pg)
    ex = {a: t.cpu().numpy() for a, t in K.rtn_export(pool, slots, dequant=True).items()}
    for s in range(n_seq):
        for p in range(n_pg):
            i = s * n_pg + p
            kp, vp = _oracle_blocks(k, v, s, p, page, k_arm, kg, vg, kbits)
            if k_arm == "rtn_token":
                assert np.array_equal(ex["k_codes"][i], O.from_matrix(kp["Q_int"], h_kv))
                assert np.array_equal(ex["k_scales"][i], O.from_matrix(kp["scale"][..., 0].astype(np.float16), h_kv))
                k16 = {"Q_int": kp["Q_int"], "scale": kp["scale"].astype(np.float16).astype(np.float32)}
            else:
                assert np.array_equal(ex["k_codes"][i], kp["Q_int"])
                assert np.array_equal(ex["k_scales"][i], kp["scale"][..., 0].astype(np.float16))
                k16 = {"Q_int": kp["Q_int"], "scale": kp["scale"].astype(np.float16).astype(np.float32)}
            assert np.array_equal(ex["v_codes"][i], O.from_matrix(vp["Q_int"], h_kv))
            assert np.array_equal(ex["v_scales"][i], O.from_matrix(vp["scale"][..., 0].astype(np.float16), h_kv))
            v16 = {"Q_int": vp["Q_int"], "scale": vp["scale"].astype(np.float16).astype(np.float32)}
            # dequant = code * (fp16-stored) scale, one float32 multiply: bit-exact
            assert np.array_equal(ex["k_deq"][i], O.dequant_packed(k_arm, k16, group=kg))
            assert np.array_equal(ex["v_deq"][i], O.dequant_packed("rtn_token", v16, group=vg))
            qmax = 2 ** (kbits - 1) - 1
            assert ex["k_codes"][i].min() >= -qmax and ex["k_codes"][i].max() <= qmax


def _decode_case(K, dev, *, page, k_arm, kg, vg, G, pages_per_seq, tail_lens, seed, h_kv=2, kbits=4):
    n_seq, max_pages, tail_cap = len(pages_per_seq), max(pages_per_seq), 256
    k, v = _inputs(seed, n_seq, h_kv, max(max_pages, 1) * page)
    g = K.rtn_geom(h_kv, G, page, k_arm, kg, vg, kbits, 2)
    n_slots = n_seq * max(max_pages, 1) + 2
    pool = K.RtnPool(g, n_slots, dev)
    gen = torch.Generator().manual_seed(seed + 1)
    table = torch.randperm(n_slots, generator=gen)[: n_seq * max(max_pages, 1)].view(n_seq, -1).to(torch.int32)
    if max_pages:
        K.rtn_append(pool, k.to(dev), v.to(dev), table.reshape(-1).contiguous().to(dev), max_pages)
    q = (torch.randn(n_seq, h_kv * G, D, generator=gen) / math.sqrt(D)).half()
    k_tail = torch.randn(n_seq, h_kv, tail_cap, D, generator=gen).half()
    v_tail = torch.randn(n_seq, h_kv, tail_cap, D, generator=gen).half()
    ws = K.rtn_workspace(g, n_seq, max_pages, dev)
    out = torch.empty(n_seq, h_kv * G, D, dtype=torch.float32, device=dev)
    scale = 1.0 / math.sqrt(D)
    K.rtn_decode(pool, q.to(dev), table.to(dev), torch.tensor(pages_per_seq, dtype=torch.int32, device=dev), max_pages,
                 k_tail.to(dev), v_tail.to(dev), torch.tensor(tail_lens, dtype=torch.int32, device=dev), scale, ws, out=out)
    torch.cuda.synchronize()
    ref = np.zeros((n_seq, h_kv * G, D), np.float32)
    for s in range(n_seq):
        kb, vb = [], []
        for p in range(pages_per_seq[s]):
            kp, vp = _oracle_blocks(k, v, s, p, page, k_arm, kg, vg, kbits)
            kp["scale"] = kp["scale"].astype(np.float16).astype(np.float32)  # the pages hold fp16 scales
            vp["scale"] = vp["scale"].astype(np.float16).astype(np.float32)
            kb.append((kp, p * page, (p + 1) * page))
            vb.append((vp, p * page, (p + 1) * page))
        tl = tail_lens[s]
        ref[s] = O.chunked_dequant_attention(
            q[s].float().numpy()[:, None, :], kb, vb, k_arm=k_arm, v_arm="rtn_token", group=kg, v_group=vg, k_pre_rope=False,
            rope_cos=None, rope_sin=None, k_tail=k_tail[s, :, :tl].float().numpy() if tl else None,
            v_tail=v_tail[s, :, :tl].float().numpy() if tl else None, n_q_groups=G, scale=scale)[:, 0, :]
    return out.cpu().numpy(), ref


def _close(out, ref, tol=2e-3):
    err, den = np.abs(out - ref).max(axis=-1), np.abs(ref).max(axis=-1)
    assert np.all(np.isfinite(out)) and np.all(err <= tol * den), f"worst relative error {float((err / den).max()):.3e}"


@pytest.mark.parametrize("page,k_arm,kg,vg,G", [(128, "rtn_channel", 32, 32, 4), (128, "rtn_token", 32, 32, 4),
                                                (64, "rtn_channel", 64, 64, 2), (64, "rtn_token", 128, 128, 8),
                                                (128, "rtn_token", 64, 32, 1)])
def test_decode_matches_oracle(page, k_arm, kg, vg, G):
    from bmx_b200 import kernels as K
    out, ref = _decode_case(K, _dev(), page=page, k_arm=k_arm, kg=kg, vg=vg, G=G, pages_per_seq=[5, 0, 3],
                            tail_lens=[37, 200, 0], seed=21)
    _close(out, ref)


def test_decode_random_geometries():
    """Sixteen geometries drawn over page, key arm, group sizes, code width, KV heads, query heads per KV head, ragged
    page counts and window lengths around the 64/128/256 edges, each against the oracle."""
    import random

    from bmx_b200 import kernels as K
    rng, dev, worst = random.Random(5), _dev(), 0.0
    for c in range(16):
        page, n_seq = rng.choice([64, 128]), rng.randint(1, 5)
        pages = [rng.choice([0, 1, 2, 3, 5, 9, 17]) for _ in range(n_seq)]
        tails = [rng.choice([0, 1, 63, 64, 65, 127, 128, 129, 255, 256]) for _ in range(n_seq)]
        tails = [max(t, 1) if p == 0 else t for p, t in zip(pages, tails)]  # a sequence holds at least one token
        cfg = dict(page=page, k_arm=rng.choice(["rtn_channel", "rtn_token"]),
                   kg=rng.choice([g for g in (32, 64, 128) if g <= page]), vg=rng.choice([32, 64, 128]),
                   G=rng.choice([1, 2, 4, 8]), pages_per_seq=pages, tail_lens=tails, seed=2000 + c,
                   h_kv=rng.choice([1, 2, 4, 8]), kbits=rng.choice([2, 3, 4]))
        out, ref = _decode_case(K, dev, **cfg)
        try:
            _close(out, ref)
        except AssertionError as e:
            raise AssertionError(f"{cfg}: {e}") from None
        worst = max(worst, float((np.abs(out - ref).max(-1) / np.abs(ref).max(-1)).max()))
    print(f"worst relative error over 16 geometries {worst:.2e}")


def test_first_baseline_config_shape():
    """Benchmark configuration 1: 8 KV heads, GQA 4, T = 4096 + 128-token window, K rtn_channel 4b, V rtn_token 2b, g = 32."""
    from bmx_b200 import kernels as K
    out, ref = _decode_case(K, _dev(), page=128, k_arm="rtn_channel", kg=32, vg=32, G=4, pages_per_seq=[32],
                            tail_lens=[128], seed=1000, h_kv=8)
    _close(out, ref)


def test_reference_golden_rtn():
    """The reference's own stacked tensors and chunked outputs (3 pages, h_kv = 2) for the same inputs."""
    from bmx_b200 import kernels as K
    dev, c = _dev(), golden("decode")
    h_kv, G, page, n_pg = 2, 4, 128, 3
    k = torch.from_numpy(O.from_matrix(c["rtn_k"], h_kv).copy())[None].half().contiguous()
    v = torch.from_numpy(O.from_matrix(c["k2b_v"], h_kv).copy())[None].half().contiguous()
    tl = c["k_tail"].shape[1]
    k_tail = torch.zeros(1, h_kv, 64, D, dtype=torch.float16)
    v_tail = torch.zeros(1, h_kv, 64, D, dtype=torch.float16)
    k_tail[0, :, :tl], v_tail[0, :, :tl] = torch.from_numpy(c["k_tail"]), torch.from_numpy(c["v_tail"])
    q = torch.from_numpy(c["q"][:, 0, :])[None].half().contiguous()
    slots = torch.arange(n_pg, dtype=torch.int32, device=dev)
    for k_arm, want in (("rtn_token", "rtn_tt_out_chunked"), ("rtn_channel", "rtn_ct_out_chunked")):
        g = K.rtn_geom(h_kv, G, page, k_arm, 32, 32, 4, 2)
        pool = K.RtnPool(g, n_pg, dev)
        K.rtn_append(pool, k.to(dev), v.to(dev), slots, n_pg)
        if k_arm == "rtn_token":
            ex = K.rtn_export(pool, slots)
            assert np.array_equal(ex["k_codes"].cpu().numpy(), c["rtn_stack_kc"])
            assert np.array_equal(ex["v_codes"].cpu().numpy(), c["rtn_stack_vc"])
            assert np.array_equal(ex["k_scales"].cpu().numpy(), c["rtn_stack_ks"])
            assert np.array_equal(ex["v_scales"].cpu().numpy(), c["rtn_stack_vs"])
        ws = K.rtn_workspace(g, 1, n_pg, dev)
        out = torch.empty(1, h_kv * G, D, dtype=torch.float32, device=dev)
        K.rtn_decode(pool, q.to(dev), slots.view(1, -1), torch.tensor([n_pg], dtype=torch.int32, device=dev), n_pg,
                     k_tail.to(dev), v_tail.to(dev), torch.tensor([tl], dtype=torch.int32, device=dev), 1.0 / math.sqrt(D), ws, out=out)
        torch.cuda.synchronize()
        _close(out.cpu().numpy(), c[want][:, 0, :][None])


@pytest.mark.parametrize("page", [64, 128])
@pytest.mark.parametrize("arm,k_group", [("rtn_channel", 32), ("rtn_channel", 64), ("rtn_channel", 128), ("rtn_token", 32), ("rtn_token", 64), ("rtn_token", 128)])
@pytest.mark.parametrize("v_group", [32, 64, 128])
def test_decode_every_kernel_variant_over_many_tiles(page, arm, k_group, v_group):
    """Each instantiation of the decode kernel with more tiles per CTA than its copy ring has stages (ranges that cross heads and
    sequences, ragged page counts, an empty sequence, a half-filled last tile), against float32 attention over the exported
    dequantized pages; queries and keys scaled by opposite powers of two must give the same attention.  Bar: 2e-3 of the largest
    output, the one of the other decode tests (fp16 rounding of the dequantized keys and of the weights, 2^-11 each)."""
    from bmx_b200 import kernels as K

    if arm == "rtn_channel" and k_group > page:
        pytest.skip("a token group never spans pages")
    dev = torch.device("cuda:0")
    h_kv, G, B, max_pages = 4, 3, 9, 61 if page == 128 else 121
    g = K.rtn_geom(h_kv, G, page, arm, k_group, v_group, 3, 2)
    gen = torch.Generator(device=dev).manual_seed(page + k_group + v_group)
    T = max_pages * page
    k = torch.randn(B, h_kv, T, 128, generator=gen, device=dev).half()
    v = torch.randn(B, h_kv, T, 128, generator=gen, device=dev).half()
    q = torch.randn(B, h_kv * G, 128, generator=gen, device=dev).half()
    table = torch.randperm(B * max_pages, generator=gen, device=dev).to(torch.int32).view(B, max_pages)
    n_pages = torch.tensor([max_pages, 1, 0, max_pages - 1, 7, 2, max_pages, 3, max_pages - 4], dtype=torch.int32, device=dev)
    k_tail, v_tail = k[:, :, :32].contiguous(), v[:, :, :32].contiguous()
    tail_len = torch.full((B,), 32, dtype=torch.int32, device=dev)
    for ks in (1.0, 2.0 ** -8, 2.0 ** 8):
        pool = K.RtnPool(g, B * max_pages, dev)
        K.rtn_append(pool, k * ks, v, table.reshape(-1).contiguous(), max_pages)
        ws = K.rtn_workspace(g, B, max_pages, dev)
        out = K.rtn_decode(pool, (q / ks).half(), table, n_pages, max_pages, (k_tail * ks).half(), v_tail, tail_len, 128 ** -0.5, ws)
        K.check_status(ws)
        ex = K.rtn_export(pool, table.reshape(-1).contiguous(), dequant=True)
        kd = ex["k_deq"].view(B, T, h_kv, 128).permute(0, 2, 1, 3)
        vd = ex["v_deq"].view(B, T, h_kv, 128).permute(0, 2, 1, 3)
        for b in range(B):
            n = int(n_pages[b]) * page
            kk = torch.cat([kd[b, :, :n], k_tail[b].float() * ks], 1)
            vv = torch.cat([vd[b, :, :n], v_tail[b].float()], 1)
            s = torch.einsum("hgd,htd->hgt", q[b].float().view(h_kv, G, 128) / ks, kk) * 128 ** -0.5
            ref = torch.einsum("hgt,htd->hgd", torch.softmax(s, -1), vv).reshape(h_kv * G, 128)
            err = float((out[b].float() - ref).abs().max() / ref.abs().max())
            assert err < 2e-3, f"scale {ks}, sequence {b}: {err:.2e}"


@pytest.mark.parametrize("arm,k_group", [("rtn_channel", 32), ("rtn_channel", 128), ("rtn_token", 32), ("rtn_token", 64)])
@pytest.mark.parametrize("kind", ["plain", "large scores", "mixed heads", "tiny keys"])
def test_decode_error_does_not_depend_on_ranges_or_other_heads(arm, k_group, kind):
    """Relative error (2-norm over all channels of a query head) against float64 attention over the exported codes and scales,
    head by head.  Two-bit keys, and four-bit keys so small that their products with the scale are multiples of 2^-24, are exact
    fp16 numbers: what is left is one fp16 rounding of each weight, 2^-11 at most.  Rounding queries times scales instead
    (9e-4 for plain two-bit keys) or scaling the queries of a group together (3e-2 for the small heads) does not stay below
    that.  "mixed heads": one head's scores pass 2^16, far beyond fp16; the others' are ordinary."""
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    h, G, B, pages = 4, 4, 2, 20
    kbits, k_scale, q_scale = {"plain": (2, 1.0, [1.0] * 4), "large scores": (2, 1.0, [3.0] * 4),
                               "mixed heads": (2, 256.0, [1024.0, 2.0 ** -8, 2.0 ** -8, 2.0 ** -10]),
                               "tiny keys": (4, 2.0 ** -16, [2.0 ** 13] * 4)}[kind]
    gen = torch.Generator(device=dev).manual_seed(1)
    channel = torch.exp(torch.randn(1, h, 1, 128, generator=gen, device=dev) * 0.7) * k_scale
    k = torch.randn(B, h, pages * 128, 128, generator=gen, device=dev) * channel  # float32: tiny keys are not fp16 numbers
    v = torch.randn(B, h, pages * 128, 128, generator=gen, device=dev)
    q = (torch.randn(B, h * G, 128, generator=gen, device=dev) * torch.tensor(q_scale, device=dev).repeat(h)[:, None]).half()
    pool = K.RtnPool(K.rtn_geom(h, G, 128, arm, k_group, 64, kbits, 2), B * pages, dev)
    table = torch.arange(B * pages, dtype=torch.int32, device=dev).view(B, pages)
    n_pages = torch.tensor([pages, pages - 3], dtype=torch.int32, device=dev)
    K.rtn_append(pool, k, v, table.reshape(-1), pages)
    ws = K.rtn_workspace(pool.geom, B, pages, dev)
    out = torch.empty(B, h * G, 128, dtype=torch.float32, device=dev)
    K.rtn_decode(pool, q, table, n_pages, pages, None, None, None, 128 ** -0.5, ws, out=out)
    K.check_status(ws)
    ex = K.rtn_export(pool, table.reshape(-1), dequant=True)
    kd, vd = (ex[n].view(B, pages * 128, h, 128).permute(0, 2, 1, 3).double() for n in ("k_deq", "v_deq"))
    for b in range(B):
        n = int(n_pages[b]) * 128
        s = torch.einsum("hgd,htd->hgt", q[b].double().view(h, G, 128), kd[b, :, :n]) * 128 ** -0.5
        want = torch.einsum("hgt,htd->hgd", torch.softmax(s, -1), vd[b, :, :n])
        err = (out[b].double().view(h, G, 128) - want).norm(dim=(0, 2)) / want.norm(dim=(0, 2))
        assert bool((err < 2.0 ** -11).all()), f"sequence {b}: {err.tolist()}"


def _rtn_codes(x, bits, group, dim):
    """Codes and float32 scales along `dim` of x (CPU float32): the reference's divisions and roundings."""
    qmax = 2 ** (bits - 1) - 1
    x = x.movedim(dim, -1)
    t = x.reshape(*x.shape[:-1], x.shape[-1] // group, group)
    am = torch.where(torch.isnan(t), torch.zeros_like(t), t.abs()).amax(-1, keepdim=True)
    scale = am.clamp_min(1e-12) / qmax
    q = torch.round(t / scale)
    q = torch.where(torch.isnan(q), torch.full_like(q, -qmax - 1), q).clamp(-qmax - 1, qmax)
    return q.reshape(x.shape).movedim(-1, dim).to(torch.int8), scale.squeeze(-1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("page,arm,k_group,v_group,kbits", [
    (128, "rtn_channel", 64, 64, 2), (128, "rtn_channel", 32, 128, 4), (128, "rtn_channel", 128, 32, 3), (128, "rtn_token", 32, 64, 4),
    (128, "rtn_token", 128, 128, 2), (64, "rtn_channel", 32, 32, 3), (64, "rtn_channel", 64, 64, 4), (64, "rtn_token", 64, 32, 2)])
@pytest.mark.parametrize("kind", ["normal", "ties", "padded", "extremes"])
def test_append_codes_equal_the_divided_ones(dtype, page, arm, k_group, v_group, kbits, kind):
    """Every code and scale of the page quantizer, whose divisions are products with the inverse scale, equals the divided one, ties,
    zeros, infinities and NaN included; also from rows that start off the sixteen-byte boundaries."""
    from bmx_b200 import kernels as K

    dev = torch.device("cuda:0")
    n, h, pages = 2, 3, 3
    T = pages * page
    gen = torch.Generator().manual_seed(page + k_group + kbits)
    k, v = torch.randn(n, h, T, 128, generator=gen), torch.randn(n, h, T, 128, generator=gen)
    if kind == "ties":  # a coarse grid: quotients fall on halves
        k, v = torch.randint(-7, 8, k.shape, generator=gen) * 0.5, torch.randint(-3, 4, v.shape, generator=gen) * 0.25
    elif kind == "padded":  # groups of nothing but zeros, of either sign, among ordinary ones
        for x in (k, v):
            x[:, :, 3::17], x[:, :, 4::17], x[..., 7], x[..., 64:96] = 0.0, -0.0, 0.0, -0.0
    elif kind == "extremes":
        for x in (k, v):
            x[:, :, 3::17] = 0
            x[:, :, 5::19] *= 1e-7
            x[:, :, 7::23] *= 3e4 if dtype == torch.float16 else 1e35
            x[0, 0, 11, 5], x[0, 1, 40, 77], x[1, 2, 70, 127] = float("inf"), float("nan"), float("-inf")
    k, v = k.to(dtype), v.to(dtype)
    g = K.rtn_geom(h, 4, page, arm, k_group, v_group, kbits, 2)
    slots = torch.arange(n * pages, dtype=torch.int32, device=dev)
    pools = [K.RtnPool(g, n * pages, dev) for _ in range(2)]
    K.rtn_append(pools[0], k.to(dev), v.to(dev), slots, pages)
    wide = torch.zeros(2, n, h, T, 128 + 3, dtype=dtype)
    wide[0, ..., 1:129], wide[1, ..., 1:129] = k, v
    wide = wide.to(dev)
    K.rtn_append(pools[1], wide[0, ..., 1:129], wide[1, ..., 1:129], slots, pages)
    assert torch.equal(pools[0].pages, pools[1].pages)
    ex = {name: t.cpu() for name, t in K.rtn_export(pools[0], slots).items()}
    kk = k.float().view(n, h, pages, page, 128).permute(0, 2, 1, 3, 4).reshape(n * pages, h, page, 128)
    vv = v.float().view(n, h, pages, page, 128).permute(0, 2, 1, 3, 4).reshape(n * pages, h, page, 128)
    vc, vs = _rtn_codes(vv, 2, v_group, 3)
    assert torch.equal(ex["v_codes"], vc) and torch.equal(ex["v_scales"].view(torch.int16), vs.half().view(torch.int16))
    if arm == "rtn_token":
        kc, ks = _rtn_codes(kk, kbits, k_group, 3)
        assert torch.equal(ex["k_codes"], kc) and torch.equal(ex["k_scales"].view(torch.int16), ks.half().view(torch.int16))
    else:
        kc, ks = _rtn_codes(kk, kbits, k_group, 2)  # codes (items, h, page, 128), scales (items, h, 128, groups)
        assert torch.equal(ex["k_codes"], kc.transpose(2, 3).reshape(n * pages, h * 128, page))
        assert torch.equal(ex["k_scales"].view(torch.int16), ks.half().reshape(n * pages, h * 128, -1).view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("page,arm,k_group,v_group,kbits", [(128, "rtn_channel", 64, 64, 2), (128, "rtn_channel", 32, 128, 4),
                                                            (128, "rtn_token", 32, 32, 3), (64, "rtn_channel", 64, 32, 4), (64, "rtn_token", 128, 64, 2)])
@pytest.mark.parametrize("tokens", [5, 700, 1290])
def test_dense_kv_equals_dequantize_and_cast(dtype, page, arm, k_group, v_group, kbits, tokens):
    """One kernel writes pages and window in the model's type: equal to dequantizing in float32, casting and concatenating."""
    from bmx_b200 import kernels as K
    from bmx_b200.engine import RtnLayerState

    dev = torch.device("cuda:0")
    B, h = 2, 3
    st = RtnLayerState(K.rtn_geom(h, 4, page, arm, k_group, v_group, kbits, 2), B, 2048, 200, dev)
    st.page_table.copy_(torch.randperm(st.page_table.numel(), device=dev).view_as(st.page_table).to(torch.int32))
    gen = torch.Generator(device=dev).manual_seed(tokens + page)
    k, v = (torch.randn(B, h, tokens, 128, generator=gen, device=dev).half() for _ in range(2))
    st.append(None, k, v)
    kd, vd = st.dense_kv(dtype)
    wk, wv = [st.k_win[:, :, : st.tail_len].to(dtype)], [st.v_win[:, :, : st.tail_len].to(dtype)]
    if st.committed:
        pk, pv = st.dense_pages()
        wk, wv = [pk.to(dtype)] + wk, [pv.to(dtype)] + wv
    assert torch.equal(kd, torch.cat(wk, 2)) and torch.equal(vd, torch.cat(wv, 2))
