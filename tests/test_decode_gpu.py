"""Decode kernels against plain PyTorch fp32 statements of the same ops."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, tol=2e-2):
    err = (got.float() - want.float()).abs().max().item()
    ref = want.float().abs().max().item() + 1e-6
    assert err / ref < tol, f"max err {err} vs {ref}"


@pytest.mark.parametrize("B", [1, 3, 8])
@pytest.mark.parametrize("N,K", [(2048, 2048), (768, 256), (2048, 1024), (512, 8192)])
def test_decode_linear_store_and_norm(B, N, K):
    from mesh_b200.ops.decode import decode_linear
    from mesh_b200.ops.norm import rmsnorm_ref
    x = torch.randn(B, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    nw = (torch.randn(K, device="cuda") * 0.1 + 1).bfloat16()
    res = torch.randn(B, N, device="cuda").bfloat16()
    y = decode_linear(x, w)
    _close(y, x.float() @ w.float().T)
    y2 = decode_linear(x, w, norm_w=nw, residual=res, out_f32=True)
    _close(y2, rmsnorm_ref(x, nw).float() @ w.float().T + res.float())


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_decode_linear_glu(act):
    from mesh_b200.ops.decode import GLU, decode_linear
    B, K, F = 4, 2048, 1024
    x = torch.randn(B, K, device="cuda").bfloat16()
    w = (torch.randn(2 * F, K, device="cuda") * 0.03).bfloat16()
    y = decode_linear(x, w, mode=GLU, act=act)
    g, u = x.float() @ w[:F].float().T, x.float() @ w[F:].float().T
    a = torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    _close(y, a * u)


@pytest.mark.parametrize("B,K,N", [(5, 2048, 1024), (1, 8192, 2048), (8, 512, 64), (3, 1024, 256), (2, 4096, 48)])
def test_decode_linear_w4(B, K, N, monkeypatch):
    """4-bit group-64 weights: the 16-byte-per-lane reader (K slices of 128 and more per warp) and the 4-byte reader
    (narrower slices, or MESH_DECODE_W4_NARROW=1) against the dequantised weights in fp32."""
    from mesh_b200.ops.decode import decode_linear, dequantize_w4, quantize_w4
    x = torch.randn(B, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.02).bfloat16()
    codes, scales = quantize_w4(w)
    wd = dequantize_w4(codes, scales)
    assert (wd.float() - w.float()).abs().max() < 0.02 * 5 / 7 + 1e-3       # half a quantisation step at 5 sigma
    y = decode_linear(x, codes, scales=scales)
    _close(y, x.float() @ wd.float().T)


@pytest.mark.parametrize("B,K,N", [(5, 2048, 1024), (1, 8192, 2048), (8, 512, 64), (3, 1024, 256)])
def test_decode_linear_w8(B, K, N):
    from mesh_b200.ops.decode import decode_linear, dequantize_w8, quantize_w8
    x = torch.randn(B, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.02).bfloat16()
    codes, scales = quantize_w8(w)
    wd = dequantize_w8(codes, scales)
    assert (wd.float() - w.float()).abs().max() < 0.02 * 5 / 127 + 5e-4
    y = decode_linear(x, codes, scales=scales)
    _close(y, x.float() @ wd.float().T)


def test_decode_glu_and_norm_with_quantised_weights():
    from mesh_b200.ops.decode import GLU, decode_linear, dequantize_w4, dequantize_w8, quantize_w4, quantize_w8
    B, K, F = 4, 2048, 512
    x = torch.randn(B, K, device="cuda").bfloat16()
    nw = (torch.randn(K, device="cuda") * 0.1 + 1).bfloat16()
    w = (torch.randn(2 * F, K, device="cuda") * 0.02).bfloat16()
    xn = (x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()).bfloat16().float()
    for quantize, dequantize in ((quantize_w4, dequantize_w4), (quantize_w8, dequantize_w8)):
        codes, scales = quantize(w)
        wd = dequantize(codes, scales).float()
        y = decode_linear(x, codes, scales=scales, norm_w=nw, eps=1e-6, mode=GLU, act="gelu_tanh")
        g, u = xn @ wd[:F].T, xn @ wd[F:].T
        _close(y, torch.nn.functional.gelu(g, approximate="tanh") * u)


def test_decode_qkv_rope_cache():
    from mesh_b200.ops.decode import QKV, decode_linear
    from mesh_b200.ops.rope import rope_ref, rope_tables
    B, K, qh, kvh, hd, S = 3, 2048, 4, 1, 256, 64
    x = torch.randn(B, K, device="cuda").bfloat16()
    w = (torch.randn((qh + 2 * kvh) * hd, K, device="cuda") * 0.03).bfloat16()
    cos, sin = rope_tables(S, hd, 1e6)
    pos = torch.tensor([5, 0, 63], dtype=torch.int32, device="cuda")
    q = torch.zeros(B, qh * hd, device="cuda", dtype=torch.bfloat16)
    kc = torch.zeros(B, kvh, S, hd, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    decode_linear(x, w, mode=QKV, qkv=dict(q_heads=qh, kv_heads=kvh, head_dim=hd, pos=pos, cos=cos, sin=sin, q_out=q,
                                           k_cache=kc, v_cache=vc, max_seq=S))
    y = (x.float() @ w.float().T)
    qr = rope_ref(y[:, :qh * hd].view(B, qh, hd), pos, cos, sin)
    kr = rope_ref(y[:, qh * hd:(qh + kvh) * hd].view(B, kvh, hd), pos, cos, sin)
    vr = y[:, (qh + kvh) * hd:].view(B, kvh, hd)
    _close(q.view(B, qh, hd), qr)
    for b in range(B):
        _close(kc[b, :, pos[b]], kr[b])
        _close(vc[b, :, pos[b]], vr[b])
    assert kc.abs().sum(-1).count_nonzero().item() == B * kvh         # only one position written per sequence


@pytest.mark.parametrize("window", [0, 16])
@pytest.mark.parametrize("T", [1, 7])
def test_decode_attention(window, T):
    from mesh_b200.ops.decode import DecodeAttention
    B, qh, kvh, hd, S = 2, 8, 2, 256, 96
    kc = torch.randn(B, kvh, S, hd, device="cuda").bfloat16()
    vc = torch.randn(B, kvh, S, hd, device="cuda").bfloat16()
    q = torch.randn(B, T, qh, hd, device="cuda").bfloat16()
    pos = torch.tensor([40, 70], dtype=torch.int32, device="cuda")
    att = DecodeAttention(B, qh, kvh, hd, splits=4, tokens_per_seq=T)
    out = torch.empty(B, T, qh * hd, device="cuda", dtype=torch.bfloat16)
    att(q, kc, vc, pos, out, window=window)
    att(q, kc, vc, pos, out, window=window)      # second launch: counters were left at zero
    for b in range(B):
        for t in range(T):
            p = int(pos[b]) + t
            lo = max(0, p - window + 1) if window else 0
            k = kc[b, :, lo:p + 1].float().repeat_interleave(qh // kvh, 0)
            v = vc[b, :, lo:p + 1].float().repeat_interleave(qh // kvh, 0)
            s = torch.einsum("hd,hkd->hk", q[b, t].float(), k) / math.sqrt(hd)
            want = torch.einsum("hk,hkd->hd", torch.softmax(s, -1), v).reshape(-1)
            _close(out[b, t], want)


def test_decode_argmax():
    from mesh_b200.ops.decode import decode_argmax
    logits = torch.randn(4, 50000, device="cuda")
    logits[2, 777] = 50.0
    logits[2, 40000] = 50.0                       # tie: lowest index wins
    tok = torch.zeros(4, dtype=torch.int32, device="cuda")
    pos = torch.zeros(4, dtype=torch.int32, device="cuda")
    step = torch.zeros(2, dtype=torch.int32, device="cuda")
    decode_argmax(logits, tok, pos, vocab_offset=1000, step=step)
    assert tok.tolist() == (logits.argmax(-1) + 1000).tolist() and tok[2].item() == 1777
    assert pos.tolist() == [1, 1, 1, 1] and step.tolist() == [1, 0]


@pytest.mark.parametrize("bits,B,K,N", [(16, 1, 256, 16), (16, 2, 768, 2384), (16, 8, 8192, 2400), (16, 5, 2560, 32), (4, 1, 1024, 48),
                                        (4, 8, 3072, 2384), (4, 3, 6144, 16), (4, 2, 1536, 64), (8, 1, 512, 16), (8, 8, 1536, 2400), (8, 3, 3072, 48)])
def test_decode_linear_streams(bits, B, K, N):
    """Short and long rings, one and several groups per CTA, odd numbers of stages.  Codes are exact inside the kernel and
    sums are fp32, so what is left is the rounding of the result: half a step of 2^-7, 2^-8 of the value at most."""
    from mesh_b200.ops.decode import decode_linear, quantize_w4, quantize_w8
    g = torch.Generator(device="cuda").manual_seed(K + N)
    x = torch.randn(B, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).bfloat16()
    if bits == 16:
        y, wd = decode_linear(x, w), w.double()
    else:
        codes, scales = (quantize_w4 if bits == 4 else quantize_w8)(w)
        if bits == 4:
            word = codes.view(torch.int32).to(torch.int64) & 0xFFFFFFFF
            c = torch.stack([(word >> (4 * n)) & 15 for n in (0, 4, 1, 5, 2, 6, 3, 7)], -1).view(N, K).double() - 8
        else:
            c = codes.double() - 128
        wd = (c.view(N, K // 64, 64) * scales.double()[..., None]).view(N, K)
        y = decode_linear(x, codes, scales=scales)
        odd = torch.empty(scales.numel() + 1, dtype=torch.float16, device="cuda")[1:].view_as(scales).copy_(scales)
        _close(decode_linear(x, codes, scales=odd), y)                    # scales off the 16-byte grid: the other reader
    want = x.double() @ wd.T
    assert float((y.double() - want).norm() / want.norm()) < 2 ** -8


@pytest.mark.parametrize("hd,qh,kvh,splits,S,window", [(256, 8, 1, 16, 300, 0), (128, 6, 2, 3, 300, 40), (64, 4, 4, 1, 64, 0),
                                                       (256, 8, 2, 64, 5000, 0), (64, 8, 1, 8, 5000, 4500)])
def test_decode_attention_clusters_and_splits(hd, qh, kvh, splits, S, window):
    """Both kernels: a cluster per KV head (few splits or a short context) and many splits merged through memory."""
    from mesh_b200.ops.decode import DecodeAttention
    B = 3
    g = torch.Generator(device="cuda").manual_seed(hd + S)
    kc, vc = (torch.randn(B, kvh, S, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(B, qh * hd, device="cuda", generator=g).bfloat16()
    pos = torch.tensor([0, S // 2, S - 1], dtype=torch.int32, device="cuda")
    att = DecodeAttention(B, qh, kvh, hd, splits=splits)
    out = torch.empty(B, qh * hd, device="cuda", dtype=torch.bfloat16)
    for _ in range(2):
        att(q, kc, vc, pos, out, window=window)
    for b in range(B):
        p = int(pos[b])
        lo = max(0, p - window + 1) if window else 0
        k, v = (t[b, :, lo:p + 1].double().repeat_interleave(qh // kvh, 0) for t in (kc, vc))
        s = torch.einsum("hd,hkd->hk", q[b].view(qh, hd).double(), k) / math.sqrt(hd)
        want = torch.einsum("hk,hkd->hd", torch.softmax(s, -1), v).reshape(-1)
        # fp32 inside, one rounding to bf16 at the end: 2^-8 of the value at most
        assert float((out[b].double() - want).norm() / want.norm()) < 2 ** -8


@pytest.mark.parametrize("V,ld", [(1, 1), (5, 8), (16383, 16384), (16384, 16384), (16385, 16385), (262144, 262144)])
def test_decode_argmax_slices(V, ld):
    from mesh_b200.ops.decode import decode_argmax
    B = 3
    logits = torch.randn(B, ld, device="cuda")[:, :V]
    logits[0, 0] = logits[0, V - 1] = 9.0                                 # tie between the first and the last slice
    logits[1, V - 1] = 9.0
    logits[2] = float("-inf")
    logits[2, V // 2] = -1e30
    tok = torch.zeros(B, dtype=torch.int32, device="cuda")
    decode_argmax(logits, tok, None)
    assert tok.tolist() == [0, V - 1, V // 2]


@pytest.mark.parametrize("V", [1, 3, 9, 33, 16388])
def test_decode_argmax_of_slices_that_take_no_time(V):
    """Few logits, or a cluster with 2056 logits for a CTA, whose pair is ready soon after it runs; every launch has other
    logits, so a pair that got lost or came from the launch before shows in the token."""
    from mesh_b200.ops.decode import decode_argmax
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(400, 8, V, device="cuda", generator=g)
    tok = torch.full((400, 8), -1, dtype=torch.int32, device="cuda")
    for i in range(400):
        decode_argmax(logits[i], tok[i], None)
    assert torch.equal(tok.long(), logits.argmax(-1))


def test_decode_linear_every_8_bit_code():
    """All 256 codes at every place of a 64-group: one input of one, so that the result is (code - 128) * scale, rounded once."""
    from mesh_b200.ops.decode import decode_linear
    K, N = 1024, 256
    place = torch.arange(K, device="cuda")
    codes = ((place[None, :] + torch.arange(N, device="cuda")[:, None]) % 256).to(torch.uint8)
    scales = torch.linspace(0.01, 2.0, N * (K // 64), device="cuda").half().view(N, K // 64)
    x = torch.zeros(8, K, device="cuda", dtype=torch.bfloat16)
    for at in (0, 1, 17, 62, 63, 500, 1023):
        x.zero_()
        x[5, at] = 1
        y = decode_linear(x, codes, scales=scales)
        want = (codes[:, at].float() - 128) * scales[:, at // 64].float()
        assert torch.equal(y[5], want.bfloat16()) and float(y[:5].abs().sum()) == 0


@pytest.mark.parametrize("bits,K,odd", [(4, 512, False), (4, 1536, False), (4, 2048, False), (8, 512, True), (8, 1536, True), (8, 2048, False)])
def test_decode_linear_codes_are_not_rounded(bits, K, odd):
    """fp32 results of both readers.  Products of integers and bf16 are exact; partial sums of 4-bit codes run on code + 128,
    up to 33 times the result: 33 * 2^-24 a step, a few steps."""
    from mesh_b200.ops.decode import decode_linear, dequantize_w4, dequantize_w8, quantize_w4, quantize_w8
    g = torch.Generator(device="cuda").manual_seed(K + bits)
    B, N = 3, 320
    x = torch.randn(B, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).bfloat16()
    codes, scales = (quantize_w4 if bits == 4 else quantize_w8)(w)
    exact = (dequantize_w4 if bits == 4 else dequantize_w8)(codes, torch.ones_like(scales)).double()
    if odd:                                                               # off the 16-byte grid: read into registers
        scales = torch.empty(scales.numel() + 1, dtype=torch.float16, device="cuda")[1:].view_as(scales).copy_(scales)
    y = decode_linear(x, codes, scales=scales, out_f32=True)
    want = x.double() @ (exact.view(N, -1, 64) * scales.double()[..., None]).view(N, K).T
    assert float((y.double() - want).norm() / want.norm()) < 2 ** -16


@pytest.mark.parametrize("bits,B,K", [(16, 8, 11776), (16, 8, 12288), (16, 8, 12800), (16, 8, 13312), (16, 8, 13568), (16, 7, 15616), (16, 6, 18176),
                                      (16, 1, 110080), (8, 8, 11264), (8, 8, 12288), (8, 8, 12800), (8, 8, 13312), (8, 7, 14336), (8, 6, 17408),
                                      (8, 1, 107520), (4, 8, 11264), (4, 8, 12288), (4, 8, 13312), (4, 7, 14336), (4, 6, 16384), (4, 1, 81920),
                                      (4, 1, 107520)])
def test_decode_linear_beside_a_large_input(bits, B, K):
    """The staged rows leave room for two stages of a ring, for two of half the size, for one, for none: every K up to what x
    and the partial sums need.  The last reader of 4-bit codes rounds weights to bf16; results are rounded to bf16."""
    from mesh_b200.ops.decode import decode_linear, dequantize_w4, dequantize_w8, quantize_w4, quantize_w8
    from mesh_b200.utils.status import check_status
    g = torch.Generator(device="cuda").manual_seed(K)
    N = 2400 if K < 20000 else 48
    x = torch.randn(B, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).bfloat16()
    if bits == 16:
        y, wd = decode_linear(x, w), w.double()
    else:
        codes, scales = (quantize_w4 if bits == 4 else quantize_w8)(w)
        y, wd = decode_linear(x, codes, scales=scales), (dequantize_w4 if bits == 4 else dequantize_w8)(codes, scales).double()
    check_status()
    want = x.double() @ wd.T
    assert float((y.double() - want).norm() / want.norm()) < 2 ** -8
    with pytest.raises(RuntimeError):                                     # beyond it the layer is refused
        decode_linear(torch.zeros(B, 16 * 8192, device="cuda", dtype=torch.bfloat16), torch.zeros(16, 16 * 8192, device="cuda", dtype=torch.bfloat16))


@pytest.mark.parametrize("bits,B,K", [(16, 8, 9216), (16, 8, 12544), (16, 6, 16640), (16, 1, 100864), (8, 6, 15360), (8, 4, 25088), (4, 5, 19456),
                                      (4, 4, 23552), (4, 1, 88064)])
def test_step_kernel_beside_a_large_input(bits, B, K):
    """A recorded step whose first layer leaves little shared memory, and a second one that reads what the first stored."""
    from mesh_b200.ops.decode import decode_linear, dequantize_w4, dequantize_w8, quantize_w4, quantize_w8, record_step
    from mesh_b200.utils.status import check_status
    g = torch.Generator(device="cuda").manual_seed(K)
    N = 3072 if K < 20000 else 1024                                       # more than one group of 16 rows for some CTAs
    x = torch.randn(B, K, device="cuda", generator=g).bfloat16()
    w, w2 = ((torch.randn(*s, device="cuda", generator=g) * 0.02).bfloat16() for s in ((N, K), (64, 512)))
    coded = (w, None) if bits == 16 else (quantize_w4 if bits == 4 else quantize_w8)(w)
    wd = w if bits == 16 else (dequantize_w4 if bits == 4 else dequantize_w8)(*coded)
    y, y2 = torch.empty(B, N, device="cuda", dtype=torch.bfloat16), torch.empty(B, 64, device="cuda", dtype=torch.bfloat16)
    with record_step() as step:
        decode_linear(x, coded[0], scales=coded[1], out=y)
        decode_linear(y[:, :512], w2, out=y2)
    for _ in range(2):
        y.zero_()
        step.run()
        check_status()
        want = x.double() @ wd.double().T
        assert float((y.double() - want).norm() / want.norm()) < 2 ** -8
        want = y[:, :512].double() @ w2.double().T
        assert float((y2.double() - want).norm() / want.norm()) < 2 ** -8


def _shifted(t, by):
    """The values of ``t`` in memory that starts ``by`` elements after an aligned address."""
    return torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)[by:].view_as(t).copy_(t)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("which,by", [("q", 1), ("k", 1), ("v", 3), ("all", 2)])
def test_decode_attention_of_inputs_at_any_address(hd, recorded, which, by):
    from mesh_b200.ops.decode import DecodeAttention, record_step
    B, qh, kvh, S = 2, 8, 2, 150
    g = torch.Generator(device="cuda").manual_seed(hd)
    kc, vc = (torch.randn(B, kvh, S, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(B, qh * hd, device="cuda", generator=g).bfloat16()
    pos = torch.tensor([S - 1, 70], dtype=torch.int32, device="cuda")
    att = DecodeAttention(B, qh, kvh, hd, splits=16)
    want, out = (torch.empty(B, qh * hd, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    att(q, kc, vc, pos, want)
    moved = [_shifted(t, by) if which in (n, "all") else t for n, t in (("q", q), ("k", kc), ("v", vc))]
    if recorded:
        with record_step() as step:
            att(*moved, pos, out)
        step.run()
    else:
        att(*moved, pos, out)
    _close(out, want, 1e-2)                                               # the same sums in another order, rounded to bf16


@pytest.mark.parametrize("at", [0, 17, 199])
@pytest.mark.parametrize("keys", [1, 200, 5000])
def test_decode_attention_keeps_a_nan(keys, at):
    """A NaN key, alone in its warp or among others, by both kernels (clusters, and 64 splits of a cache of 5000): the heads that
    read it are NaN, the others are not."""
    from mesh_b200.ops.decode import DecodeAttention
    qh, kvh, hd = 8, 2, 128
    at = min(at, keys - 1)
    g = torch.Generator(device="cuda").manual_seed(keys)
    kc, vc = (torch.randn(1, kvh, max(keys, 256), hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    kc[0, 1, at, 5] = float("nan")
    q = torch.randn(1, qh * hd, device="cuda", generator=g).bfloat16()
    pos = torch.tensor([keys - 1], dtype=torch.int32, device="cuda")
    out = torch.empty(1, qh * hd, device="cuda", dtype=torch.bfloat16)
    DecodeAttention(1, qh, kvh, hd, splits=64)(q, kc, vc, pos, out)
    assert torch.isnan(out.view(qh, hd)).all(-1).tolist() == [False] * 4 + [True] * 4 and not torch.isnan(out.view(qh, hd)[:4]).any()
