"""tcgen05 flash attention forward vs an fp32 PyTorch statement: causal, sliding window, GQA, head dims, offsets/strides."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, tol=2e-2):
    err = (got.float() - want.float()).abs().max().item()
    ref = want.float().abs().max().item() + 1e-6
    assert err / ref < tol, f"max err {err} vs {ref}"


@pytest.mark.parametrize("hd,H,Hkv", [(128, 4, 4), (256, 8, 2), (64, 2, 1)])
@pytest.mark.parametrize("Tq,Tk,causal,window", [(256, 256, True, 0), (384, 384, True, 100), (200, 330, False, 0), (512, 512, True, 512)])
def test_flash_forward(hd, H, Hkv, Tq, Tk, causal, window):
    from mesh_b200.ops.attention import attention_ref, flash_attention
    from mesh_b200.utils.status import check_status
    B = 2
    q = torch.randn(B, Tq, H, hd, device="cuda").bfloat16()
    k = torch.randn(B, Tk, Hkv, hd, device="cuda").bfloat16()
    v = torch.randn(B, Tk, Hkv, hd, device="cuda").bfloat16()
    out, lse = flash_attention(q, k, v, causal=causal, window=window, need_lse=True)
    check_status()
    ref, lse_ref = attention_ref(q, k, v, causal, window)
    _close(out, ref)
    torch.testing.assert_close(lse, lse_ref, atol=2e-2, rtol=2e-2)


def test_flash_fused_qkv_view_and_striped_positions():
    from mesh_b200.ops.attention import attention_ref, flash_attention, merge_partials
    B, T, H, Hkv, hd = 1, 256, 4, 2, 128
    qkv = torch.randn(B, T, (H + 2 * Hkv) * hd, device="cuda").bfloat16()
    q = qkv[..., :H * hd].view(B, T, H, hd)
    k = qkv[..., H * hd:(H + Hkv) * hd].view(B, T, Hkv, hd)
    v = qkv[..., (H + Hkv) * hd:].view(B, T, Hkv, hd)
    out = flash_attention(q, k, v, causal=True)
    _close(out, attention_ref(q, k, v, True)[0])
    # two striped halves of the keys merged by log-sum-exp equal attention over all keys
    o_full, _ = attention_ref(q, k, v, True)
    parts = []
    for r in range(2):
        parts.append(flash_attention(q, k[:, r::2].contiguous(), v[:, r::2].contiguous(), causal=True, k_off=r, k_stride=2, need_lse=True))
    o, _ = merge_partials(parts[0][0], parts[0][1], parts[1][0], parts[1][1])
    _close(o, o_full)


def _ring_rank(rank, world, rdv, striped, overlap=False):
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.ops.attention import attention_ref, ring_attention
    from mesh_b200.utils.status import check_status
    torch.cuda.set_device(rank)
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(rank, world, torch.device("cuda", rank), rdv, None)
    B, T, H, hd = 1, 256 * world, 4, 128
    g = torch.Generator(device="cpu").manual_seed(0)
    q, k, v = (torch.randn(B, T, H, hd, generator=g).bfloat16().cuda() for _ in range(3))
    sl = slice(rank, T, world) if striped else slice(rank * (T // world), (rank + 1) * (T // world))
    o, _ = ring_attention(q[:, sl].contiguous(), k[:, sl].contiguous(), v[:, sl].contiguous(), ctx.comm, causal=True,
                          striped=striped, overlap=overlap)
    torch.cuda.synchronize()
    check_status()
    ref, _ = attention_ref(q, k, v, True)
    _close(o, ref[:, sl])
    rdv.barrier("ring-done")
    ctx.heap.close()


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("striped", [False, True])
def test_ring_attention_two_ranks(striped, overlap):
    """``overlap``: the next KV chunk travels on a side stream under the attention of the current one."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    from mesh_b200.utils.launch import spawn_ranks
    spawn_ranks(_ring_rank, 2, striped, overlap, use_cuda=True, timeout=300.0)


def _ref_grads(q, k, v, dout, causal, window):
    from mesh_b200.ops.attention import attention_ref
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    o, _ = attention_ref(qf, kf, vf, causal, window)
    o.backward(dout.float())
    return qf.grad, kf.grad, vf.grad


@pytest.mark.parametrize("hd,H,Hkv", [(128, 4, 4), (128, 4, 2), (64, 2, 1), (256, 4, 2)])
@pytest.mark.parametrize("T,causal,window", [(256, True, 0), (384, True, 100), (200, False, 0)])
def test_flash_backward(hd, H, Hkv, T, causal, window):
    """Head size 256 has the forward kernel and a backward in blocks of tensor operations; 64 and 128 both kernels."""
    from mesh_b200.ops.attention import attention
    from mesh_b200.utils.status import check_status
    torch.manual_seed(1)
    B = 2
    q = torch.randn(B, T, H, hd, device="cuda").bfloat16().requires_grad_(True)
    k = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16().requires_grad_(True)
    v = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16().requires_grad_(True)
    dout = torch.randn(B, T, H, hd, device="cuda").bfloat16()
    out = attention(q, k, v, causal=causal, window=window)
    out.backward(dout)
    torch.cuda.synchronize()
    check_status()
    dq, dk, dv = _ref_grads(q.detach(), k.detach(), v.detach(), dout, causal, window)
    _close(q.grad, dq, 3e-2)
    _close(k.grad, dk, 3e-2)
    _close(v.grad, dv, 3e-2)


def _ring_bwd_rank(rank, world, rdv, striped):
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.ops.attention import ring_attention_autograd
    from mesh_b200.utils.status import check_status
    torch.cuda.set_device(rank)
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(rank, world, torch.device("cuda", rank), rdv, None)
    B, T, H, Hkv, hd = 1, 256 * world, 4, 2, 128
    g = torch.Generator(device="cpu").manual_seed(0)
    q = torch.randn(B, T, H, hd, generator=g).bfloat16().cuda()
    k, v = (torch.randn(B, T, Hkv, hd, generator=g).bfloat16().cuda() for _ in range(2))
    dout = torch.randn(B, T, H, hd, generator=g).bfloat16().cuda()
    sl = slice(rank, T, world) if striped else slice(rank * (T // world), (rank + 1) * (T // world))
    ql, kl, vl = (t[:, sl].contiguous().requires_grad_(True) for t in (q, k, v))
    o = ring_attention_autograd(ql, kl, vl, ctx.comm, causal=True, striped=striped)
    o.backward(dout[:, sl].contiguous())
    torch.cuda.synchronize()
    check_status()
    dq, dk, dv = _ref_grads(q, k, v, dout, True, 0)
    _close(ql.grad, dq[:, sl], 3e-2)
    _close(kl.grad, dk[:, sl], 3e-2)
    _close(vl.grad, dv[:, sl], 3e-2)
    rdv.barrier("ring-bwd-done")
    ctx.heap.close()


@pytest.mark.parametrize("striped", [False, True])
def test_ring_attention_backward_two_ranks(striped):
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    from mesh_b200.utils.launch import spawn_ranks
    spawn_ranks(_ring_bwd_rank, 2, striped, use_cuda=True, timeout=300.0)


def _ulysses_rank(rank, world, rdv):
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.ops.attention import ulysses_attention
    from mesh_b200.parallel.topology import AxisContext
    from mesh_b200.utils.status import check_status
    torch.cuda.set_device(rank)
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(rank, world, torch.device("cuda", rank), rdv, None)
    axis = AxisContext("cp", rank, list(range(world)), ctx.device, None, ctx.heap)
    B, T, H, Hkv, hd = 1, 256 * world, 4, 2, 128
    g = torch.Generator(device="cpu").manual_seed(0)
    q = torch.randn(B, T, H, hd, generator=g).bfloat16().cuda()
    k, v = (torch.randn(B, T, Hkv, hd, generator=g).bfloat16().cuda() for _ in range(2))
    dout = torch.randn(B, T, H, hd, generator=g).bfloat16().cuda()
    sl = slice(rank * (T // world), (rank + 1) * (T // world))
    ql, kl, vl = (t[:, sl].contiguous().requires_grad_(True) for t in (q, k, v))
    o = ulysses_attention(ql, kl, vl, axis, causal=True)
    o.backward(dout[:, sl].contiguous())
    torch.cuda.synchronize()
    check_status()
    dq, dk, dv = _ref_grads(q, k, v, dout, True, 0)
    from mesh_b200.ops.attention import attention_ref
    ref, _ = attention_ref(q, k, v, True)
    _close(o, ref[:, sl])
    _close(ql.grad, dq[:, sl], 3e-2)
    _close(kl.grad, dk[:, sl], 3e-2)
    _close(vl.grad, dv[:, sl], 3e-2)
    rdv.barrier("ulysses-done")
    ctx.heap.close()


def test_head_exchange_attention_two_ranks():
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    from mesh_b200.utils.launch import spawn_ranks
    spawn_ranks(_ulysses_rank, 2, use_cuda=True, timeout=300.0)


@pytest.mark.parametrize("hd,H,Hkv,T,causal", [(128, 4, 2, 256, True), (64, 2, 2, 200, False), (256, 2, 1, 256, True)])
def test_flash_forward_with_dropout_matches_the_logical_mask(hd, H, Hkv, T, causal):
    """Dropout inside the kernel: Philox keyed by (head, query position, key position), against the fp32 statement
    that applies the same mask; the kept fraction is 1 - p."""
    from mesh_b200.ops.attention import attention_ref, flash_attention
    from mesh_b200.ops.philox import attention_keep_mask
    from mesh_b200.utils.status import check_status
    torch.manual_seed(3)
    B = 2
    q = torch.randn(B, T, H, hd, device="cuda").bfloat16()
    k = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16()
    v = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16()
    drop = dict(p=0.25, seed=0x1234_5678_9ABC, site=3, execution=7)
    out = flash_attention(q, k, v, causal=causal, dropout=drop)
    check_status()
    ref, _ = attention_ref(q, k, v, causal, dropout=drop)
    _close(out, ref, 3e-2)
    plain, _ = attention_ref(q, k, v, causal)
    assert (out.float() - plain).abs().max() > 0.05                  # the mask did something
    keep = attention_keep_mask(torch.zeros(1, 1, dtype=torch.int64), torch.arange(512)[:, None], torch.arange(512)[None, :],
                               0.25, drop["seed"], drop["site"], drop["execution"])
    assert abs(float(keep.float().mean()) - 0.75) < 0.01


def test_dropout_is_the_same_for_a_shard_of_the_queries_and_of_the_heads():
    from mesh_b200.ops.attention import flash_attention
    torch.manual_seed(4)
    B, T, H, hd = 1, 512, 4, 128
    q, k, v = (torch.randn(B, T, H, hd, device="cuda").bfloat16() for _ in range(3))
    drop = dict(p=0.3, seed=99)
    whole = flash_attention(q, k, v, causal=True, dropout=drop)
    # the second half of the queries, as a sequence shard would hold them (logical positions through q_off)
    part = flash_attention(q[:, 256:].contiguous(), k, v, causal=True, q_off=256, dropout=drop)
    _close(part, whole[:, 256:], 1e-2)                                 # another mask would differ by O(1)
    # heads 2..3 only, as a tensor-parallel rank would hold them
    heads = flash_attention(q[:, :, 2:].contiguous(), k[:, :, 2:].contiguous(), v[:, :, 2:].contiguous(), causal=True,
                            dropout=dict(drop, head_off=2, heads_total=4))
    _close(heads, whole[:, :, 2:], 1e-2)


@pytest.mark.parametrize("hd,H,Hkv", [(128, 4, 2), (64, 2, 2)])
def test_flash_backward_with_dropout(hd, H, Hkv):
    from mesh_b200.ops.attention import attention, attention_ref
    from mesh_b200.utils.status import check_status
    torch.manual_seed(5)
    B, T = 2, 256
    q = torch.randn(B, T, H, hd, device="cuda").bfloat16().requires_grad_(True)
    k = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16().requires_grad_(True)
    v = torch.randn(B, T, Hkv, hd, device="cuda").bfloat16().requires_grad_(True)
    dout = torch.randn(B, T, H, hd, device="cuda").bfloat16()
    drop = dict(p=0.2, seed=77, site=1)
    attention(q, k, v, causal=True, dropout=drop).backward(dout)
    check_status()
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    o, _ = attention_ref(qf, kf, vf, True, dropout=drop)
    o.backward(dout.float())
    _close(q.grad, qf.grad, 3e-2)
    _close(k.grad, kf.grad, 3e-2)
    _close(v.grad, vf.grad, 3e-2)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,H,Hkv,causal,window,off,stride", [
    (1, 1, 1, 1, 1, True, 0, (0, 0), 1),             # a single key: its output is v, its score gradients vanish
    (2, 129, 129, 2, 1, True, 0, (0, 0), 1),         # one row past a tile
    (1, 257, 257, 4, 2, True, 1, (0, 0), 1),         # a window of one key
    (2, 383, 640, 2, 2, False, 0, (0, 0), 1),        # ragged ends, several key blocks
    (1, 700, 700, 4, 1, True, 130, (0, 0), 1),       # the window moves the first key block of the two query tiles apart
    (1, 512, 512, 2, 2, True, 0, (1, 0), 2),         # striped positions
    (1, 300, 512, 2, 2, True, 0, (0, 150), 1),       # queries that see no key
])
def test_flash_tiles(hd, B, Tq, Tk, H, Hkv, causal, window, off, stride):
    """Both directions at the edges of the query tiles and key blocks, every row by itself.  A row's probabilities, score
    gradients and results are rounded to bf16, 2^-9 of their size at most each: three of them stay below 8e-3 of the row.
    Delta is formed from the rounded output; dP - Delta cancels where few keys are seen, so the rounding that is left of it,
    three standard deviations of sum(dO o O), is allowed on the rows of dq and dk that it reaches."""
    from mesh_b200.ops.attention import flash_attention, flash_attention_backward
    from mesh_b200.utils.status import check_status
    g = torch.Generator(device="cuda").manual_seed(3)
    q, do = (torch.randn(B, Tq, H, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Tk, Hkv, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    kw = dict(causal=causal, window=window, q_off=off[0], q_stride=stride, k_off=off[1], k_stride=stride)
    out, lse = flash_attention(q, k, v, need_lse=True, **kw)
    dq, dk, dv = flash_attention_backward(q, k, v, out, lse, do, **kw)
    check_status()
    qf, kf, vf = (t.double().requires_grad_(True) for t in (q, k, v))
    s = torch.einsum("bthd,bshd->bhts", qf, kf.repeat_interleave(H // Hkv, 2)) * hd ** -0.5
    qp, kp = off[0] + torch.arange(Tq, device="cuda") * stride, off[1] + torch.arange(Tk, device="cuda") * stride
    hide = torch.zeros(Tq, Tk, dtype=torch.bool, device="cuda")
    if causal:
        hide |= kp[None] > qp[:, None]
    if window:
        hide |= kp[None] <= qp[:, None] - window
    s = s.masked_fill(hide, float("-inf"))
    blind = hide.all(-1)
    pr = torch.softmax(s.masked_fill(blind[:, None], 0.0), -1).masked_fill(blind[:, None], 0.0)
    ref = torch.einsum("bhts,bshd->bthd", pr, vf.repeat_interleave(H // Hkv, 2))
    grads = torch.autograd.grad(ref, (qf, kf, vf), do.double())
    with torch.no_grad():
        left = 3 * 2 ** -9 * hd ** -0.5 * (do.double() * ref).square().sum(-1).sqrt()                    # [B, Tq, H]
        left_q = left * torch.einsum("bhts,bshd->bthd", pr, kf.repeat_interleave(H // Hkv, 2)).norm(dim=-1)
        left_k = torch.einsum("bhts,bth->bsh", pr.square(), (left * qf.norm(dim=-1)).square())
        left_k = left_k.view(B, Tk, Hkv, H // Hkv).sum(-1).sqrt()
        for name, got, want, extra in (("out", out, ref, 0.0), ("dq", dq, grads[0], left_q), ("dk", dk, grads[1], left_k), ("dv", dv, grads[2], 0.0)):
            err, limit = (got.double() - want).norm(dim=-1), 8e-3 * want.norm(dim=-1) + extra + 1e-6
            worst = int((err / limit).argmax())
            assert bool((err <= limit).all()), (name, worst, float(err.view(-1)[worst]), float(limit.view(-1)[worst]))
    seen = ~blind
    torch.testing.assert_close(lse[:, :, seen].double(), torch.logsumexp(s, -1)[:, :, seen].detach(), atol=1e-4, rtol=1e-4)
    assert bool(torch.isinf(lse[:, :, blind]).all())


@pytest.mark.parametrize("B,T,Hq,Hkv,hd,window", [(2, 200, 4, 2, 64, 0), (1, 257, 2, 2, 128, 100), (3, 64, 4, 1, 256, 0)])
def test_rotary_attention_of_a_fused_projection(B, T, Hq, Hkv, hd, window):
    """Against the separate rotation and attention with the same kernels' oracles; the projection may be a column slice."""
    from mesh_b200.ops.attention import attention_ref, rotary_attention
    from mesh_b200.ops.rope import rope_tables
    from mesh_b200.utils.status import check_status
    g = torch.Generator(device="cuda").manual_seed(B * T)
    W = (Hq + 2 * Hkv) * hd
    wide = torch.randn(B * T, W + 64, device="cuda", generator=g).bfloat16()
    qkv = wide[:, 32:32 + W].requires_grad_(True)
    do = torch.randn(B, T, Hq, hd, device="cuda", generator=g).bfloat16()
    cos, sin = rope_tables(2 * T, hd, 1e4)
    pos = (torch.arange(B * T, device="cuda", dtype=torch.int32) % T) * 2
    out = rotary_attention(qkv, pos, cos, sin, batch=B, q_heads=Hq, kv_heads=Hkv, head_dim=hd, window=window)
    (d,) = torch.autograd.grad(out, qkv, do)
    check_status()
    x = qkv.detach().float().requires_grad_(True)
    m = x.view(B * T, Hq + 2 * Hkv, hd)
    c, s = cos[pos.long()][:, None], sin[pos.long()][:, None]
    lo, hi = m[:, :Hq + Hkv, :hd // 2], m[:, :Hq + Hkv, hd // 2:]
    r = torch.cat([lo * c - hi * s, hi * c + lo * s], -1).view(B, T, Hq + Hkv, hd)
    ref, _ = attention_ref(r[:, :, :Hq], r[:, :, Hq:], m[:, Hq + Hkv:].view(B, T, Hkv, hd), True, window)
    (dref,) = torch.autograd.grad(ref, x, do.float())
    # rotated heads, probabilities, score gradients and results are rounded to bf16: 2^-9 each on average, four of them
    assert float((out.float() - ref).norm() / ref.norm()) < 8e-3
    assert float((d.float() - dref).norm() / dref.norm()) < 8e-3


@pytest.mark.parametrize("p", [0.0, 0.1])
@pytest.mark.parametrize("T", [100, 256, 300, 640, 901])
def test_flash_heads_of_256_alternate_between_groups(T, p):
    """One to eight key blocks, with and without the (slow) dropout draws in between, several times: the groups of warps
    meet in every order."""
    from mesh_b200.ops.attention import attention_ref, flash_attention
    from mesh_b200.utils.status import check_status
    B, H, Hkv, hd = 2, 4, 2, 256
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, n, hd, device="cuda", generator=g).bfloat16() for n in (H, Hkv, Hkv))
    kw = dict(causal=True, window=0 if T < 600 else 300, dropout=dict(p=p, seed=7) if p else None)
    ref, lse_ref = attention_ref(q, k, v, **kw)
    for _ in range(4):
        out, lse = flash_attention(q, k, v, need_lse=True, **kw)
        # probabilities and results are rounded to bf16
        assert float((out.float() - ref).norm() / ref.norm()) < 6e-3
        torch.testing.assert_close(lse, lse_ref, atol=1e-4, rtol=1e-4)
    check_status()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (1, 5, 3), (3, 333, 5), (2, 4097, 7)])
def test_delta_of_any_number_of_rows(hd, B, T, H):
    """Row sums of dO o O, from fewer rows than a warp holds to more than the grid takes at once, with the accumulator cleared."""
    from mesh_b200.ops.attention import _delta
    g = torch.Generator(device="cuda").manual_seed(T)
    do, o = (torch.randn(B, T, H, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    clear = torch.full((B, T, H, hd), float("nan"), device="cuda")
    got = _delta(do, o, clear)
    want = (do.double() * o.double()).sum(-1).transpose(1, 2)
    # fp32 sums of hd products of order one
    assert float((got.double() - want).abs().max()) < hd * 2 ** -20
    assert float(clear.abs().sum()) == 0


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("T", [40, 100, 200, 256])
@pytest.mark.parametrize("p", [0.0, 0.1])
def test_a_sample_does_not_reach_the_one_before_it(hd, T, p):
    """The last tile of a sample ends in rows of the next one.  A sample of NaN or infinities changes nothing in the others."""
    from mesh_b200.ops.attention import flash_attention, flash_attention_backward
    from mesh_b200.utils.status import check_status
    g = torch.Generator(device="cuda").manual_seed(T)
    clean = dict(zip("qkvd", (torch.randn(3, T, 2, hd, device="cuda", generator=g).bfloat16() for _ in range(4))))
    kw = dict(causal=False, dropout=dict(p=p, seed=5) if p else None)

    def run(t):
        out, lse = flash_attention(t["q"], t["k"], t["v"], need_lse=True, **kw)
        grads = flash_attention_backward(t["q"], t["k"], t["v"], *fixed, t["d"], **kw) if hd < 256 else ()
        return out, lse, *grads

    fixed = flash_attention(clean["q"], clean["k"], clean["v"], need_lse=True, **kw)
    want = run(clean)
    for name in "qkvd":
        for value in (float("nan"), float("inf")):
            bad = dict(clean, **{name: clean[name].clone()})
            bad[name][1] = value
            for got, ref in zip(run(bad), want):
                for b in (0, 2):
                    assert bool(torch.isfinite(got[b]).all()), (name, value, b)
                    # the same products; only the order in which blocks of dq are added may differ
                    torch.testing.assert_close(got[b], ref[b], atol=1e-4, rtol=1e-4)
    check_status()
