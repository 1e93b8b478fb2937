"""The work a program does through this library, as cases that can be timed and checked.

A case is one layer's call on a packed KV cache: quantize pages into the pool (a prompt prefix, or the page per sequence that
a streaming step commits), one decode step over pages and window, or the attention of a block of prompt rows.  The codecs are
the library's: "k2b" (low-rank keys + 3-bit residual, Hadamard + 2-bit values), "rtn" (plain groupwise rounding, the kivi
recipe among it) and "spectral" (per-head K4 key packs).  Head geometry, window, rotary base, ranks, groups and context
lengths are those of the benchmark, the recipes and the tests.

`exact` restates the codecs and the attention in float64 with plain torch, from the same seeded inputs.
"""

import math
from types import SimpleNamespace

import torch

from bmx_b200 import kernels as K
from bmx_b200.engine import K2bLayerState, RtnLayerState, SpectralLayerState
from bmx_b200.packed_streaming import PackedStreamingLayer
from bmx_b200.recipes import spec_pair
from bmx_b200.rope import default_rope_tables

D = 128
WINDOW = 128          # recent tokens kept in fp16
THETA = 5e5           # rotary base of the benchmark's model shape
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
# directions per bit width of a spectral pack: 104 of 128 with bits (2.6 bits per direction), and a leaner table
TIERS = {"wide": {8: 2, 6: 6, 5: 10, 4: 16, 3: 26, 2: 44}, "lean": {6: 2, 5: 6, 4: 14, 3: 22, 2: 36}}
LLOYD = (-1.5194618701934814, -0.46033763885498047, 0.44421979784965515, 1.5017313957214355)  # 2-bit levels of N(0, 1)

HEADS = {"h_kv": 8, "q_groups": 4}
K2B = {**HEADS, "page": 128, "rank": 32, "group": 64, "shared_basis": False}
RTN = {**HEADS, "page": 128, "k_arm": "rtn_channel", "kbits": 4, "k_group": 32, "v_group": 32}
KIVI = {**HEADS, "page": 128, "k_arm": "rtn_channel", "kbits": 2, "k_group": 64, "v_group": 64}
SPECTRAL = {**HEADS, "group": 64, "tiers": "wide"}


def listed():
    return [
        # the first tokens of a reply to a short prompt, one user: launches and latency
        {"name": "k2b_decode_b1_t2048", "kind": "k2b_decode", "batch": 1, "tokens": 2048 + 128, **K2B, "rank": 16},
        # the benchmark's step: eight sequences of 32k tokens
        {"name": "k2b_decode_b8_t32768", "kind": "k2b_decode", "batch": 8, "tokens": 32768 + 128, **K2B},
        # 64-token pages, one basis over all heads, an odd length and an odd batch
        {"name": "k2b_decode_b3_t9001_page64", "kind": "k2b_decode", "batch": 3, "tokens": 9001, **K2B, "page": 64, "rank": 16, "group": 32,
         "shared_basis": True},
        # the page that each of sixteen sequences commits once in 128 decode steps
        {"name": "k2b_append_b16_p1", "kind": "k2b_append", "batch": 16, "pages": 1, "dtype": "f16", **K2B},
        # prompts of 16k tokens enter the cache
        {"name": "k2b_append_b4_p128", "kind": "k2b_append", "batch": 4, "pages": 128, "dtype": "bf16", **K2B},
        # a follow-up turn of 512 tokens over a 16k-token conversation
        {"name": "k2b_prefill_b1_n512_t16384", "kind": "k2b_prefill", "batch": 1, "rows": 512, "tokens": 16384 + 128, **K2B},
        # the last block of a prompt that is taken in blocks of 2048 rows, two prompts at once
        {"name": "k2b_prefill_b2_n2048_t8192", "kind": "k2b_prefill", "batch": 2, "rows": 2048, "tokens": 8192 + 128, **K2B},
        # prompts of 16k tokens enter a plain RTN cache (kivi)
        {"name": "rtn_append_b4_p128", "kind": "rtn_append", "batch": 4, "pages": 128, "dtype": "f16", **KIVI},
        # a decode step of sixteen sequences over it
        {"name": "rtn_decode_b16_t8192", "kind": "rtn_decode", "batch": 16, "tokens": 8192 + 128, **RTN},
        # a prompt block of 1024 rows over 8k tokens under the kivi recipe, as the model's attention function calls it
        {"name": "rtn_prompt_b1_n1024_t8192", "kind": "rtn_prompt", "batch": 1, "rows": 1024, "tokens": 8192 + 128, "dtype": "bf16", **KIVI},
        # prompts of 8k tokens enter a spectral cache (keys and values)
        {"name": "spectral_append_b4_p64", "kind": "spectral_append", "batch": 4, "pages": 64, "dtype": "f16", **SPECTRAL},
        # a decode step of 32 sequences over it
        {"name": "spectral_decode_b32_t8192", "kind": "spectral_decode", "batch": 32, "tokens": 8192 + 128, **SPECTRAL},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["k2b_decode", "k2b_append", "k2b_prefill", "rtn_append", "rtn_decode", "rtn_prompt", "spectral_append", "spectral_decode"])
    heads = {"h_kv": rng.choice([2, 3, 4, 8]), "q_groups": rng.choice([1, 2, 4, 8])}
    case = {"kind": kind, **heads}
    if kind.startswith("k2b"):
        page = 128 if kind == "k2b_prefill" else rng.choice([128, 128, 64])
        case.update(page=page, rank=rng.choice([16, 32]), group=rng.choice([g for g in (32, 64, 128) if page % g == 0]),
                    shared_basis=rng.random() < 0.4)
    elif kind.startswith("rtn"):
        group = rng.choice([32, 64, 128])
        case.update(page=128, k_arm=rng.choice(["rtn_channel", "rtn_token"]), kbits=rng.choice([2, 3, 4]), k_group=group, v_group=group)
    else:
        case.update(group=rng.choice([32, 64, 128]), tiers=rng.choice(sorted(TIERS)))
    if kind.endswith("decode"):
        case["tokens"] = _log(rng, 300, 32768) if kind == "k2b_decode" else _log(rng, 300, 12000)
        most = {"k2b_decode": 8 * 32768, "rtn_decode": 16 * 8192, "spectral_decode": 32 * 8192}[kind]
        case["batch"] = _log(rng, 1, max(1, min(32, most // case["tokens"])))
    elif kind.endswith("append"):
        case["pages"] = _log(rng, 1, 128 if kind != "spectral_append" else 64)
        case["batch"] = _log(rng, 1, max(1, min(16, (512 if kind != "spectral_append" else 256) // case["pages"])))
        case["dtype"] = rng.choice(["f16", "bf16", "f32"])
    else:
        case["rows"] = _log(rng, 2, 2048 if kind == "k2b_prefill" else 1024)
        case["tokens"] = case["rows"] + _log(rng, 300, 16384 - case["rows"] if kind == "k2b_prefill" else 7000)
        case["batch"] = rng.choice([1, 2]) if case["rows"] * case["tokens"] <= 2048 * 8192 and kind == "k2b_prefill" else 1
        if kind == "rtn_prompt":
            case["dtype"] = rng.choice(["f16", "bf16"])
    return case


# ---- seeded inputs -----------------------------------------------------------------------------------------------------


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _n_tokens(case):
    return case["tokens"] if "tokens" in case else case["pages"] * case.get("page", 128)


def _committed(case):
    """Tokens held as packed pages: whole pages beyond the recent window."""
    S, page = case["tokens"], case.get("page", 128)
    return (S - WINDOW) // page * page if S > WINDOW else 0


def _rotation(gen, n, rank=D):
    out = []
    for _ in range(n):
        Q, R = torch.linalg.qr(torch.randn(D, rank, generator=gen, device=gen.device))
        out.append(Q * torch.sign(torch.diagonal(R)))
    return torch.stack(out)


def _k2b_basis(case, gen):
    """(h_kv * 128, rank) float32: one orthonormal basis per head, or one over all heads (the heads' bases side by side)."""
    per_head = _rotation(gen, case["h_kv"], case["rank"])
    b = per_head.reshape(case["h_kv"] * D, case["rank"])
    return (b / math.sqrt(case["h_kv"]) if case["shared_basis"] else b).contiguous()


def _k2b_kv(case, gen, basis, dtype):
    """Pre-RoPE keys: a low-rank signal with a falling spectrum plus noise; values N(0, 1)."""
    B, h, T, r = case["batch"], case["h_kv"], _n_tokens(case), case["rank"]
    decay = torch.arange(1, r + 1, device=gen.device).float() ** -1.5
    heads = basis.view(h, D, r) * (math.sqrt(h) if case["shared_basis"] else 1.0)
    if case["shared_basis"]:
        coef = (torch.randn(B, 1, T, r, generator=gen, device=gen.device) * decay).expand(B, h, T, r)
    else:
        coef = torch.randn(B, h, T, r, generator=gen, device=gen.device) * decay
    k = torch.matmul(coef, heads.transpose(1, 2))
    k = (k + 0.1 * torch.randn(B, h, T, D, generator=gen, device=gen.device)).to(dtype)
    v = torch.randn(B, h, T, D, generator=gen, device=gen.device).to(dtype)
    return k, v


def _rtn_kv(case, gen, dtype):
    """Post-RoPE keys with channel scales that differ by an order of magnitude (why kivi groups along tokens); values N(0, 1)."""
    B, h, T = case["batch"], case["h_kv"], _n_tokens(case)
    scale = torch.exp(torch.randn(1, h, 1, D, generator=gen, device=gen.device) * 0.7)
    k = (torch.randn(B, h, T, D, generator=gen, device=gen.device) * scale).to(dtype)
    return k, torch.randn(B, h, T, D, generator=gen, device=gen.device).to(dtype)


def _spectral_inputs(case, gen, dtype):
    """Orthogonal per-head encoders, a power-law spectrum, bit widths by variance rank; keys drawn from that spectrum."""
    B, h, T = case["batch"], case["h_kv"], _n_tokens(case)
    enc = _rotation(gen, h)
    by_rank = [b for b in sorted(TIERS[case["tiers"]], reverse=True) for _ in range(TIERS[case["tiers"]][b])]
    by_rank += [0] * (D - len(by_rank))
    perm = torch.stack([torch.randperm(D, generator=gen, device=gen.device) for _ in range(h)])
    bits = torch.zeros(h, D, dtype=torch.int64, device=gen.device)
    bits.scatter_(1, perm, torch.tensor(by_rank, device=gen.device).expand(h, D))
    lam = torch.zeros(h, D, device=gen.device)
    lam.scatter_(1, perm, (torch.arange(1, D + 1, device=gen.device).float() ** -1.2).expand(h, D))
    y = torch.randn(B, h, T, D, generator=gen, device=gen.device) * (lam.sqrt() * 4.0)[None, :, None, :]
    k = torch.matmul(y, enc.transpose(1, 2)).to(dtype)
    v = torch.randn(B, h, T, D, generator=gen, device=gen.device).to(dtype)
    return enc, bits, k, v


def _rope(x, cos, sin):
    return x * cos + torch.cat((-x[..., D // 2:], x[..., :D // 2]), -1) * sin


def _queries(case, gen, dtype=torch.float16):
    shape = (case["batch"], case["h_kv"] * case["q_groups"], case["rows"], D) if "rows" in case else (case["batch"], case["h_kv"] * case["q_groups"], D)
    return torch.randn(*shape, generator=gen, device=gen.device).to(dtype)


def _causal_mask(case, device):
    S, n = case["tokens"], case["rows"]
    return torch.ones(n, S, dtype=torch.bool, device=device).tril(S - n)[None, None]


def prepare(case, seed):
    kind, gen, dev = case["kind"], _gen(seed), _device()
    B, h, G = case["batch"], case["h_kv"], case["q_groups"]
    s = {"case": case}
    if kind in ("k2b_decode", "k2b_prefill"):
        basis = _k2b_basis(case, gen)
        k, v = _k2b_kv(case, gen, basis, torch.float16)
        cos, sin = (t.half() for t in default_rope_tables(THETA, D, case["tokens"] + 256, device=dev))
        geom = K.k2b_geom(h, G, case["page"], case["rank"], case["group"], 1 if case["shared_basis"] else h)
        st = K2bLayerState(geom, B, case["tokens"], WINDOW, dev, cos, sin)
        st.set_basis(basis)
        T = case["tokens"]
        st.append(k, _rope(k, cos[:T], sin[:T]), v)
        s.update(state=st, q=_queries(case, gen))
    elif kind == "k2b_append":
        basis = _k2b_basis(case, gen)
        k, v = _k2b_kv(case, gen, basis, DTYPES[case["dtype"]])
        geom = K.k2b_geom(h, G, case["page"], case["rank"], case["group"], 1 if case["shared_basis"] else h)
        n = B * case["pages"]
        s.update(k=k, v=v, basis=basis, pool=K.K2bPool(geom, n, dev), slots=torch.arange(n, dtype=torch.int32, device=dev))
    elif kind in ("rtn_append", "rtn_decode"):
        geom = K.rtn_geom(h, G, case["page"], case["k_arm"], case["k_group"], case["v_group"], case["kbits"], 2)
        k, v = _rtn_kv(case, gen, DTYPES[case.get("dtype", "f16")])
        if kind == "rtn_append":
            n = B * case["pages"]
            s.update(k=k, v=v, pool=K.RtnPool(geom, n, dev), slots=torch.arange(n, dtype=torch.int32, device=dev))
        else:
            st = RtnLayerState(geom, B, case["tokens"], WINDOW, dev)
            st.append(None, k, v)
            s.update(state=st, q=_queries(case, gen))
    elif kind == "rtn_prompt":
        k_spec, v_spec = spec_pair("kivi", group=case["k_group"])
        k_spec.arm, k_spec.bits = case["k_arm"], case["kbits"]
        config = SimpleNamespace(num_attention_heads=h * G, num_key_value_heads=h, head_dim=D, hidden_size=h * G * D,
                                 max_position_embeddings=32768, rope_theta=THETA, rope_parameters={"rope_type": "default", "rope_theta": THETA},
                                 standardize_rope_params=lambda: None)  # the fields of a model's config that the layer reads
        layer = PackedStreamingLayer(k_spec, v_spec, config, recent_window=WINDOW)
        k, v = _rtn_kv(case, gen, torch.float16)
        with torch.no_grad():
            layer.update(k, v)
        s.update(layer=layer, q=_queries(case, gen, DTYPES[case["dtype"]]), mask=_causal_mask(case, dev))
    else:
        enc, bits, k, v = _spectral_inputs(case, gen, DTYPES[case.get("dtype", "f16")])
        pack = K.SpectralPackDev(enc.cpu(), enc.cpu(), bits.cpu(), page=128, group=case["group"], device=dev)
        if kind == "spectral_append":
            n = B * case["pages"]
            s.update(pack=pack, k=k, v=v, kpool=pack.new_pool(n), vpool=K.vblock_pool(h, n, dev), slots=torch.arange(n, dtype=torch.int32, device=dev))
        else:
            cos, sin = (t.half() for t in default_rope_tables(THETA, D, case["tokens"] + 256, device=dev))
            T = case["tokens"]
            st = SpectralLayerState(pack, G, B, T, WINDOW, dev, cos, sin)
            st.append(k, _rope(k, cos[:T], sin[:T]), v)
            s.update(state=st, q=_queries(case, gen))
    if kind in ("k2b_append", "spectral_append"):
        s.update(signs=K.hadamard_signs(D, 0).to(dev), codebook=torch.tensor(LLOYD, dtype=torch.float32, device=dev))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind.endswith("_decode"):
        return s["state"].decode(s["q"])
    if kind == "k2b_prefill":
        return s["state"].prefill_attend(s["q"], case["tokens"] - case["rows"])
    if kind == "rtn_prompt":
        return s["layer"].attend(s["q"], 1.0 / math.sqrt(D), is_causal=True, attention_mask=s["mask"])
    if kind == "k2b_append":
        K.k2b_append(s["pool"], s["k"], s["v"], s["basis"], s["signs"], s["codebook"], s["slots"], case["pages"])
        return {"pages": s["pool"].pages, "coefs": s["pool"].coefs}
    if kind == "rtn_append":
        K.rtn_append(s["pool"], s["k"], s["v"], s["slots"], case["pages"])
        return {"pages": s["pool"].pages}
    K.spectral_append(s["pack"], s["kpool"], s["k"], s["slots"], case["pages"])
    K.vblock_append(s["vpool"], s["v"], s["signs"], s["codebook"], s["slots"], case["pages"])
    return {"keys": s["kpool"], "values": s["vpool"]}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------


def _bytes_per_token_head(case):
    """Packed bytes of one token of one KV head (codes, scales, norms, coefficients)."""
    kind = case["kind"]
    if kind.startswith("k2b"):
        coef = 2 * case["rank"] / (case["h_kv"] if case["shared_basis"] else 1)
        return coef + D / 2 + 2 * D / case["group"] + D / 4 + 2
    if kind.startswith("rtn"):
        k_scale = 2 * D / case["k_group"]  # per channel and token group, or per token and channel group: the same count
        return D / 2 + k_scale + D / 4 + 2 * D / case["v_group"]
    code_bits = sum(n * (2 if b == 2 else 4 if b <= 4 else 8) for b, n in TIERS[case["tiers"]].items())
    used = sum(TIERS[case["tiers"]].values())
    return code_bits / 8 + 4 * used / case["group"] + D / 4 + 2


def work(case):
    kind, B, h, G = case["kind"], case["batch"], case["h_kv"], case["q_groups"]
    packed = _bytes_per_token_head(case)
    used = sum(TIERS[case["tiers"]].values()) if "tiers" in case else 0
    # operations per token and KV head besides attention: the products that make or undo the key code, the value rotation
    code_ops = {"k2b": 2 * D * case.get("rank", 0), "rtn": 0, "spe": 2 * D * used}[kind[:3]]
    if kind.endswith("append"):
        units = B * h * _n_tokens(case)
        ops = {"k2b": 2 * code_ops + 7 * D, "rtn": 0, "spe": 2 * D * used + 7 * D}[kind[:3]] + 4 * D
        return {"bytes": units * (2 * D * DTYPES[case["dtype"]].itemsize + packed), "flops": units * ops}
    S, done = case["tokens"], _committed(case)
    n_q = case.get("rows", 1)
    bytes_ = B * h * (done * packed + (S - done) * 2 * D * 2) + 2 * B * h * G * n_q * D * 2
    visible = n_q * (S - n_q) + n_q * (n_q + 1) // 2  # (row, key) pairs under the causal mask; S for one row
    return {"bytes": bytes_, "flops": B * h * (done * code_ops + visible * G * 4 * D)}


def tolerance(case):
    """Packed bytes are whole values and have to be the same.  Attention outputs are fp16 (bf16 under a bf16 model) results of
    fp16 products: about four times what a pass differs from the float64 restatement, which is 8e-4 for k2b and spectral
    pages and 2.2e-3 for RTN pages (larger scores), 7e-3 with keys, values and output in bf16."""
    if case["kind"].endswith("append"):
        return "exact"
    if case.get("dtype") == "bf16":
        return {"rel": 2.5e-2}
    return {"rel": 9e-3 if case["kind"].startswith("rtn") else 3e-3}


# ---- float64 restatement -----------------------------------------------------------------------------------------------


def _hadamard():
    H = torch.ones(1, 1, dtype=torch.float64, device=_device())
    while H.shape[0] < D:
        H = torch.cat([torch.cat([H, H], 1), torch.cat([H, -H], 1)], 0)
    return H / math.sqrt(D)


def _values_back(v):
    """Hadamard + 2-bit Lloyd round trip of (..., 128) values: fp16 norm, nearest level, inverse rotation."""
    g = torch.Generator().manual_seed(0)
    signs = (torch.randint(0, 2, (D,), generator=g) * 2 - 1).to(v.device, torch.float64)
    lev = torch.tensor(LLOYD, dtype=torch.float64, device=v.device)
    x = v.double()
    norm = x.norm(dim=-1, keepdim=True).clamp_min(1e-12).half().double()
    y = (x / norm * signs) @ _hadamard() * math.sqrt(D)
    idx = torch.bucketize(y, (lev[1:] + lev[:-1]) / 2)
    return (lev[idx] / math.sqrt(D)) @ _hadamard() * signs * norm


def _rtn_back(x, bits, group, dim):
    """Symmetric groupwise rounding of x along `dim`, scales stored as fp16."""
    qmax = 2 ** (bits - 1) - 1
    x = x.double().movedim(dim, -1)
    t = x.reshape(*x.shape[:-1], x.shape[-1] // group, group)
    scale = t.abs().amax(-1, keepdim=True).clamp_min(1e-12) / qmax
    t = torch.round(t / scale).clamp(-qmax - 1, qmax) * scale.half().double()
    return t.reshape(x.shape).movedim(-1, dim)


def _keys_back(case, seq_k, extra):
    """Committed keys (h, T, 128) of one sequence after the codec's round trip, before rotation."""
    x = seq_k.double()
    if case["kind"].startswith("rtn"):
        return _rtn_back(x, case["kbits"], case["k_group"], 1 if case["k_arm"] == "rtn_channel" else 2)
    if case["kind"].startswith("k2b"):
        h, T, _ = x.shape
        r = case["rank"]
        b = extra.double()
        if case["shared_basis"]:
            us = (x.permute(1, 0, 2).reshape(T, h * D) @ b).half().double()
            low = (us @ b.half().double().T).view(T, h, D).permute(1, 0, 2)
        else:
            bh = b.view(h, D, r)
            low = torch.matmul(torch.matmul(x, bh).half().double(), bh.half().double().transpose(1, 2))
        return low + _rtn_back(x - low, 3, case["group"], 1)
    enc, bits = extra
    y = torch.matmul(x, enc.double())                      # (h, T, 128)
    h, T, _ = y.shape
    t = y.transpose(1, 2).reshape(h, D, T // case["group"], case["group"])
    b = bits.double()[:, :, None, None]
    qmax = 2.0 ** (b - 1) - 1
    qmax = torch.where(b > 0, qmax, torch.ones_like(qmax))
    scale = t.abs().amax(-1, keepdim=True).clamp_min(1e-12) / qmax

    def codes(sc):
        return torch.minimum(torch.maximum(torch.round(t / sc), -qmax - 1), qmax)

    for _ in range(10):
        q = codes(scale)
        scale = ((t * q).sum(-1, keepdim=True) / (q * q).sum(-1, keepdim=True).clamp_min(1e-12)).clamp_min(1e-12)
    y_hat = torch.where(b > 0, codes(scale) * scale, torch.zeros_like(t)).reshape(h, D, T).transpose(1, 2)
    return torch.matmul(y_hat, enc.double().transpose(1, 2))


def exact(case, seed):
    """What `run` returns, in float64.  The appends return packed bytes in this library's own order: no computed numbers."""
    kind = case["kind"]
    if kind.endswith("append"):
        return None
    gen = _gen(seed)
    if kind.startswith("k2b"):
        extra = _k2b_basis(case, gen)
        k, v = _k2b_kv(case, gen, extra, torch.float16)
    elif kind.startswith("rtn"):
        extra = None
        k, v = _rtn_kv(case, gen, torch.float16)
    else:
        enc, bits, k, v = _spectral_inputs(case, gen, torch.float16)
        extra = (enc, bits)
    q = _queries(case, gen, DTYPES[case.get("dtype", "f16")])
    S, done, h, G = case["tokens"], _committed(case), case["h_kv"], case["q_groups"]
    rotated = not kind.startswith("rtn")
    if rotated:  # the tables are inputs: fp16, as the caches keep them
        inv = 1.0 / (THETA ** (torch.arange(0, D, 2, dtype=torch.int64, device=k.device).float() / D))
        fr = torch.arange(S, device=k.device).float()[:, None] * inv[None, :]
        cos, sin = torch.cat((fr, fr), -1).cos().half(), torch.cat((fr, fr), -1).sin().half()
    n_q = case.get("rows", 1)
    pos = torch.arange(S - n_q, S, device=k.device)
    out = []
    for b in range(case["batch"]):
        kd, vd = k[b].double(), v[b].double()
        if rotated:
            kd = _rope(k[b], cos, sin).double()            # the window holds the model's own rotated keys
        if done:
            back = _keys_back(case, k[b, :, :done], extra)
            kd[:, :done] = _rope(back, cos[:done].double(), sin[:done].double()) if rotated else back
            vd[:, :done] = _values_back(v[b, :, :done]) if rotated else _rtn_back(v[b, :, :done], 2, case["v_group"], 2)
        qb = q[b].double().view(h, G, n_q, D)
        rows = []
        for r0 in range(0, n_q, 256):                      # bounded score matrices
            sc = torch.einsum("hgnd,htd->hgnt", qb[:, :, r0:r0 + 256], kd) / math.sqrt(D)
            sc = sc.masked_fill(torch.arange(S, device=k.device)[None, :] > pos[r0:r0 + 256, None], float("-inf"))
            rows.append(torch.einsum("hgnt,htd->hgnd", torch.softmax(sc, -1), vd))
        out.append(torch.cat(rows, 2).reshape(h * G, n_q, D))
    out = torch.stack(out)
    return out if "rows" in case else out[:, :, 0]
