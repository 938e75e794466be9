"""RMSNorm, RoPE and router top-k kernels against fp32 PyTorch statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 2048), (7, 1536), (300, 4096), (64, 8192)])
def test_rmsnorm_fwd(rows, cols):
    from mesh_b200.ops.norm import rmsnorm_fwd, rmsnorm_ref
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    w = (torch.randn(cols, device="cuda") * 0.1 + 1).bfloat16()
    y, _, _ = rmsnorm_fwd(x, w, 1e-6)
    torch.testing.assert_close(y.float(), rmsnorm_ref(x, w).float(), atol=2e-2, rtol=2e-2)
    r = torch.randn(rows, cols, device="cuda").bfloat16()
    y2, res, _ = rmsnorm_fwd(x, w, 1e-6, residual=r, weight_offset=1.0)
    s = (x.float() + r.float()).bfloat16()
    torch.testing.assert_close(res.float(), s.float(), atol=1e-2, rtol=1e-2)
    torch.testing.assert_close(y2.float(), rmsnorm_ref(s, w, weight_offset=1.0).float(), atol=3e-2, rtol=3e-2)


def test_rmsnorm_bwd():
    from mesh_b200.ops.norm import rmsnorm
    x = torch.randn(500, 2048, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(2048, device="cuda") * 0.1 + 1).bfloat16().requires_grad_(True)
    dy = torch.randn(500, 2048, device="cuda").bfloat16()
    rmsnorm(x, w).backward(dy)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    yr.backward(dy.float())
    torch.testing.assert_close(x.grad.float(), xr.grad, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.5, rtol=3e-2)


@pytest.mark.parametrize("heads,hd", [(8, 256), (16, 128), (2, 64)])
def test_rope(heads, hd):
    from mesh_b200.ops.rope import rope_, rope_ref, rope_tables
    T = 77
    cos, sin = rope_tables(1024, hd, theta=1e6)
    pos = torch.randint(0, 1024, (T,), device="cuda", dtype=torch.int32)
    x = torch.randn(T, heads, hd, device="cuda").bfloat16()
    want = rope_ref(x, pos, cos, sin)
    got = rope_(x.clone(), pos, cos, sin)
    torch.testing.assert_close(got.float(), want.float(), atol=2e-2, rtol=2e-2)
    back = rope_(got.clone(), pos, cos, sin, inverse=True)
    torch.testing.assert_close(back.float(), x.float(), atol=4e-2, rtol=4e-2)


@pytest.mark.parametrize("E,k", [(64, 6), (8, 2), (256, 8), (40, 3)])
def test_router_topk(E, k):
    from mesh_b200.ops.router import router_topk, router_topk_ref
    T = 1000
    logits = torch.randn(T, E, device="cuda")
    bias = torch.randn(E, device="cuda")
    w, i = router_topk(logits, k, bias)
    wr, ir = router_topk_ref(logits, k, bias)
    assert torch.equal(i, ir)
    torch.testing.assert_close(w, wr, atol=1e-5, rtol=1e-4)


@pytest.mark.parametrize("n", [8, 1000, 4096 * 512, 4096 * 4096 + 3])
def test_dot_sum(n):
    from mesh_b200.ops.loss import dot_sum
    a = torch.randn(n, device="cuda").bfloat16()
    b = torch.randn(n, device="cuda").bfloat16()
    for _ in range(2):                     # the second call finds the scratch as the first left it
        got = dot_sum(a, b)
    want = (a.double() * b.double()).sum()
    assert abs(float(got) - float(want)) <= 1e-3 * float((a.double() * b.double()).abs().sum().sqrt()) + 1e-3


@pytest.mark.parametrize("n,v,start", [(64, 1000, 0), (300, 25152, 25152), (7, 4099, 100)])
def test_cross_entropy_kernels_match_fp32(n, v, start):
    """One vocabulary shard alone (group of one): loss and gradient against torch's fp32 cross-entropy over the shard,
    with targets outside the shard and ignored rows."""
    from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
    torch.manual_seed(0)
    logits = (torch.randn(n, v, device="cuda") * 3).bfloat16().requires_grad_(True)
    targets = torch.randint(start, start + v, (n,), device="cuda")
    targets[::5] = -100
    loss = vocab_parallel_cross_entropy(logits, targets, start, None, reduction="sum")
    loss.backward()
    ref = logits.detach().float().requires_grad_(True)
    local = torch.where(targets == -100, targets, targets - start)
    want = torch.nn.functional.cross_entropy(ref, local, ignore_index=-100, reduction="sum")
    want.backward()
    assert abs(float(loss) - float(want)) <= 2e-3 * abs(float(want)) + 1e-3
    assert float((logits.grad.float() - ref.grad).abs().max()) < 8e-3


@pytest.mark.parametrize("n,v,ld,reduction", [(1, 1, 1, "mean"), (5, 7, 9, "none"), (3, 16384 + 9, 16384 + 9, "mean"), (1300, 2049, 2056, "sum"),
                                              (4, 4096, 8192, "mean")])
def test_cross_entropy_rows_of_any_alignment(n, v, ld, reduction):
    """Rows that start off the 16-byte grid, a row stride that differs from the width, masked logits (-inf), all rows
    ignored but one, targets in the first, the last and no column's vector body; losses in fp32 (relative 1e-5), gradients
    rounded to bf16 (2^-8)."""
    from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
    g = torch.Generator(device="cuda").manual_seed(v)
    buf = (torch.randn(n, ld, device="cuda", generator=g) * 3).bfloat16()
    logits = buf[:, :v].detach()
    if v > 8:
        logits[:, 2:5] = float("-inf")
    logits.requires_grad_(True)
    t = torch.tensor([0, v - 1, v // 2 if v > 16 else 0], device="cuda").repeat(-(-n // 3))[:n].contiguous()
    if n > 3:
        t[1:] = torch.where(torch.arange(1, n, device="cuda") % 4 == 0, -100, t[1:])
    loss = vocab_parallel_cross_entropy(logits, t, 0, None, reduction=reduction)
    up = torch.rand(loss.shape, device="cuda", generator=g) + 0.5
    (d,) = torch.autograd.grad(loss, logits, up)
    ref = logits.detach().double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(ref, t, ignore_index=-100, reduction=reduction)
    (dw,) = torch.autograd.grad(want, ref, up.double())
    torch.testing.assert_close(loss.double(), want.detach(), rtol=1e-5, atol=1e-5)
    # p - 1 cancels in the target's column: its error is fp32's of p (1e-6 of the upstream value)
    assert bool(((d.double() - dw).abs() <= 2 ** -8 * dw.abs() + 2e-6 * float(up.max())).all())


@pytest.mark.parametrize("v", [4096, 4099])
@pytest.mark.parametrize("off", [0.0, 100.0, -1000.0, 60000.0])
def test_cross_entropy_of_logits_far_from_zero(off, v):
    """The loss depends on the differences of the logits alone.  fp32: exponents below 20 are within 2^-20, the logarithm of a
    sum within as much; gradients are rounded to bf16, and in the target's column p - 1 cancels."""
    from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
    g = torch.Generator(device="cuda").manual_seed(v)
    n = 33
    logits = (torch.randn(n, v, device="cuda", generator=g) * 4 + off).bfloat16().requires_grad_(True)
    t = torch.randint(0, v, (n,), device="cuda", generator=g)
    t[0] = logits[0].argmax()
    loss = vocab_parallel_cross_entropy(logits, t, 0, None, reduction="none")
    (d,) = torch.autograd.grad(loss.sum(), logits)
    ref = logits.detach().double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(ref, t, reduction="none")
    (dw,) = torch.autograd.grad(want.sum(), ref)
    # the largest difference of two logits here is 512 (a bf16 step at 60000 is 256): the loss is rounded at that size
    spread = float((ref.amax(-1) - ref.amin(-1)).max().detach())
    torch.testing.assert_close(loss.double(), want.detach(), rtol=2 ** -22, atol=2 ** -23 * max(20.0, spread))
    assert bool(((d.double() - dw).abs() <= 2 ** -8 * dw.abs() + 2e-6).all())


@pytest.mark.parametrize("masked", ["start", "row", "all but one", "alternating"])
@pytest.mark.parametrize("v", [40, 8192, 8195])
def test_cross_entropy_of_logits_masked_with_the_lowest_value(v, masked):
    """Finite masks (bf16's lowest value) over whole vectors, over what a thread reads first, and over whole rows."""
    from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
    g = torch.Generator(device="cuda").manual_seed(v)
    low = torch.finfo(torch.bfloat16).min
    logits = (torch.randn(3, v, device="cuda", generator=g) * 3).bfloat16()
    if masked == "start":
        logits[:, :v // 2] = low
    elif masked == "row":
        logits[1] = low
    elif masked == "all but one":
        logits[:, :-1] = low
    else:
        logits.view(-1)[::2] = low
    logits.requires_grad_(True)
    t = torch.tensor([v - 1, v - 2, v - 1], device="cuda")
    loss = vocab_parallel_cross_entropy(logits, t, 0, None, reduction="none")
    (d,) = torch.autograd.grad(loss.sum(), logits)
    ref = logits.detach().double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(ref, t, reduction="none")
    (dw,) = torch.autograd.grad(want.sum(), ref)
    torch.testing.assert_close(loss.double(), want.detach(), rtol=1e-5, atol=1e-5)
    assert bool(((d.double() - dw).abs() <= 2 ** -8 * dw.abs() + 2e-6).all())


@pytest.mark.parametrize("v,at", [(1, 0), (7, 3), (17, 0), (17, 16), (300, 2), (4099, 4098), (4099, 1)])
@pytest.mark.parametrize("rest", ["finite", "-inf"])
def test_cross_entropy_keeps_a_nan(v, at, rest):
    """Wherever the NaN logit lies (before the first 16-byte boundary, in the vectors, after them) and whether or not a thread
    has seen a finite value before it."""
    from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
    buf = torch.randn(3 * v + 1, device="cuda").bfloat16()[1:].view(3, v)      # rows at odd addresses
    if rest == "-inf":
        buf[1] = float("-inf")
    buf[1, at] = float("nan")
    t = torch.full((3,), (at + 1) % v, device="cuda")
    loss = vocab_parallel_cross_entropy(buf, t, 0, None, reduction="none")
    assert torch.isnan(loss).tolist() == [False, True, False]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rmsnorm_backward_of_no_rows(dtype):
    """The weight gradient of an empty batch is zero, in memory that held something else."""
    from mesh_b200.ops.norm import rmsnorm_bwd
    cols = 2048
    x, w = torch.empty(0, cols, device="cuda", dtype=torch.bfloat16), torch.ones(cols, device="cuda", dtype=torch.bfloat16)
    rstd = torch.empty(0, device="cuda")
    for _ in range(4):
        junk = [torch.full((cols,), float("nan"), dtype=dtype, device="cuda") for _ in range(8)]
        del junk
        dx, dw = rmsnorm_bwd(x, x, w, rstd, 0.0, dtype)
        assert dx.shape == x.shape and dw.dtype == dtype and float(dw.abs().sum()) == 0
    from ctypes import c_float, c_int, c_void_p
    from mesh_b200 import _native
    dw = torch.full((cols,), float("nan"), device="cuda")
    p = lambda t: c_void_p(t.data_ptr())
    assert _native.lib().mesh_rmsnorm_bwd_noalloc(p(x), p(x), p(w), p(rstd), p(x), p(dw), c_int(0), c_int(cols), c_float(0.0),
                                                  c_void_p(_native.stream())) == 0
    assert float(dw.abs().sum()) == 0
