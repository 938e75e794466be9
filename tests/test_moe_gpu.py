"""Expert-parallel MoE layer (fused dispatch / grouped tcgen05 GEMMs / combine) vs a dense fp32 PyTorch statement."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, tol):
    err = (got.float() - want.float()).abs().max().item()
    ref = want.float().abs().max().item() + 1e-6
    assert err / ref < tol, f"max err {err} vs {ref}"


def _run(rank, world, rdv, T, D, F, E, k, steps):
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.parallel.moe import EPMoE, moe_reference
    from mesh_b200.utils.status import check_status
    torch.cuda.set_device(rank)
    dev = torch.device("cuda", rank)
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(rank, world, dev, rdv, None)
    g = torch.Generator(device="cpu").manual_seed(0)
    xs = [torch.randn(T, D, generator=g).bfloat16() for _ in range(world)]
    dys = [torch.randn(T, D, generator=g).bfloat16() for _ in range(world)]
    wr = (torch.randn(E, D, generator=g) * 0.1).bfloat16()
    w1 = (torch.randn(E, 2 * F, D, generator=g) * 0.05).bfloat16()
    w2 = (torch.randn(E, D, F, generator=g) * 0.05).bfloat16()
    bias = [torch.randn(E, generator=g) for _ in range(world)]          # per-rank bias: skewed, uneven loads
    El = E // world
    moe = EPMoE(ctx, T, D, F, E, k, capacity_factor=3.0)
    x, dy = xs[rank].to(dev), dys[rank].to(dev)
    w1l = w1[rank * El:(rank + 1) * El].reshape(El * 2 * F, D).contiguous().to(dev)
    w2l = w2[rank * El:(rank + 1) * El].reshape(El * D, F).contiguous().to(dev)
    wrd, bd = wr.to(dev), bias[rank].to(dev)
    for _ in range(steps):
        out = moe.forward(x, wrd, w1l, w2l, bd)
        dx, dwr, dw1, dw2 = moe.backward(dy)
    check_status()
    assert int(moe.layout[3 * El + 1]) == 0, "capacity overflow in the test configuration"
    # reference: all ranks' tokens through all experts, autograd for the gradients
    W1, W2, WR = w1.to(dev).float().requires_grad_(True), w2.to(dev).float().requires_grad_(True), wr.to(dev).float().requires_grad_(True)
    outs, xrs = [], []
    for r in range(world):
        xr = xs[r].to(dev).float().requires_grad_(True)
        outs.append(moe_reference(xr, WR, W1, W2, k, bias[r].to(dev)))
        xrs.append(xr)
    sum((o * dys[r].to(dev).float()).sum() for r, o in enumerate(outs)).backward()
    _close(out, outs[rank], 3e-2)
    _close(dx, xrs[rank].grad, 5e-2)
    _close(dw1.view(El, 2 * F, D), W1.grad[rank * El:(rank + 1) * El], 5e-2)
    _close(dw2.view(El, D, F), W2.grad[rank * El:(rank + 1) * El], 5e-2)
    rdv.barrier("moe-done")
    ctx.heap.close()


def test_moe_world1():
    import torch.distributed as dist
    from mesh_b200.runtime.rendezvous import Rendezvous
    _run(0, 1, Rendezvous(dist.HashStore(), 0, 1), 256, 256, 128, 8, 2, 2)


@pytest.mark.parametrize("world", [2, 4, 8])
def test_moe_expert_parallel(world):
    if torch.cuda.device_count() < world:
        pytest.skip(f"needs {world} GPUs")
    from mesh_b200.utils.launch import spawn_ranks
    spawn_ranks(_run, world, 256, 256, 128, 8 * world // 2 if world > 2 else 8, 2, 2, use_cuda=True, timeout=300.0)


@pytest.mark.parametrize("T,D,F,E,k,spread", [(64, 256, 128, 8, 8, 0.0), (192, 512, 256, 16, 12, 6.0), (320, 256, 384, 64, 1, 4.0)])
def test_moe_unused_experts_and_many_choices(T, D, F, E, k, spread):
    """More choices than are read together, experts that no token chose (their weight gradients are zero, in memory that
    held something else), and the router's gradient, against the dense statement's autograd."""
    import torch.distributed as dist
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.parallel.moe import EPMoE, moe_reference
    from mesh_b200.runtime.rendezvous import Rendezvous
    from mesh_b200.utils.status import check_status
    dev = torch.device("cuda", 0)
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(0, 1, dev, Rendezvous(dist.HashStore(), 0, 1), None)
    g = torch.Generator(device=dev).manual_seed(5)
    rand = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=dev) * std).bfloat16()
    x, dy, wr, w1, w2 = rand(T, D), rand(T, D), rand(E, D, std=0.02), rand(E, 2 * F, D, std=0.05), rand(E, D, F, std=0.05)
    bias = torch.linspace(spread, -spread, E, device=dev)                # the last experts are chosen by nobody
    moe = EPMoE(ctx, T, D, F, E, k, capacity_factor=2.0)
    torch.full((E * 3 * F * D * 2,), float("nan"), dtype=torch.bfloat16, device=dev)       # what freed memory may hold
    out = moe.forward(x, wr, w1.view(-1, D), w2.view(-1, F), bias)
    dx, dwr, dw1, dw2 = moe.backward(dy)
    check_status()
    X, W1, W2, WR = (t.float().requires_grad_(True) for t in (x, w1, w2, wr))
    want = moe_reference(X, WR, W1, W2, k, bias)
    # the statement routes on rounded logits, whose rounding autograd passes straight through
    gx, g1, g2, gr = torch.autograd.grad((want * dy.float()).sum(), (X, W1, W2, WR), allow_unused=True)
    unused = (moe.layout[:E] == 0)
    if spread:
        assert bool(unused.any())
    assert float(dw1.view(E, 2 * F, D)[unused].abs().sum()) == 0 and float(dw2.view(E, D, F)[unused].abs().sum()) == 0
    for got, ref in ((out, want), (dx, gx), (dw1.view_as(g1), g1), (dw2.view_as(g2), g2)):
        _close(got.float(), ref.detach(), 4e-2)
    if k > 1:
        _close(dwr, gr, 4e-2)
    else:                                             # one renormalised weight is the constant 1
        assert float(dwr.abs().max()) < 1e-4
    ctx.heap.close()


def test_plan_whose_counts_never_come():
    """Every CTA of the planning kernel gives up on the counts of a step that nobody counted: the tables are empty, the status
    says why, and the layer works again afterwards."""
    import ctypes
    import torch.distributed as dist
    from mesh_b200 import _native
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.parallel import moe as moe_module
    from mesh_b200.runtime.rendezvous import Rendezvous
    from mesh_b200.utils.status import MeshDeviceError, check_status, status_block
    dev = torch.device("cuda", 0)
    set_config(MeshConfig.from_env(heap_bytes=256 << 20))
    ctx = MeshContext(0, 1, dev, Rendezvous(dist.HashStore(), 0, 1), None)
    T, D, F, E, k = 128, 256, 128, 16, 2
    g = torch.Generator(device=dev).manual_seed(1)
    rand = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=dev) * std).bfloat16()
    x, wr, w1, w2 = rand(T, D), rand(E, D, std=0.1), rand(E * 2 * F, D, std=0.05), rand(E * D, F, std=0.05)
    moe = moe_module.EPMoE(ctx, T, D, F, E, k)
    want = moe.forward(x, wr, w1, w2).clone()
    lengths = moe.n_tiles.tolist()
    assert all(n > 0 for n in lengths[:6]) and lengths[6:] == [0, 0]
    p = moe_module._Plan()
    p.counts, p.seq, p.rank, p.world, p.experts = moe.counts.ptr(), moe.steps + 1, 0, 1, E
    p.cap_rows, p.d_model, p.d_ff = moe.cap, D, F
    p.send_base, p.layout = moe.send_base.data_ptr(), moe.layout.data_ptr()
    for i in range(6):
        p.tables[i] = moe.tables[i].data_ptr()
    p.n_tiles, p.max_tiles, p.status = moe.n_tiles.data_ptr(), moe.max_tiles, status_block(dev).data_ptr()
    _native.check(moe.L.mesh_moe_plan(ctypes.byref(p), moe_module._s()), "mesh_moe_plan")
    assert moe.n_tiles.tolist() == [0] * 8
    with pytest.raises(MeshDeviceError):
        check_status()
    assert torch.equal(moe.forward(x, wr, w1, w2), want) and moe.n_tiles.tolist() == lengths
    check_status()
    ctx.heap.close()


@pytest.mark.parametrize("F,E", [(64, 16), (192, 16), (320, 8)])
def test_moe_experts_of_any_height(F, E):
    """2 F is not a multiple of a 256-row tile: the last tile of an expert's gate and up gradient ends inside it, and stays out
    of the next expert's rows, whatever order the tiles finish in."""
    import torch.distributed as dist
    from mesh_b200.config import MeshConfig, set_config
    from mesh_b200.distributed.context import MeshContext
    from mesh_b200.parallel.moe import EPMoE, moe_reference
    from mesh_b200.runtime.rendezvous import Rendezvous
    from mesh_b200.utils.status import check_status
    dev = torch.device("cuda", 0)
    T, D, k = 256, 512, 2
    set_config(MeshConfig.from_env(heap_bytes=512 << 20))
    ctx = MeshContext(0, 1, dev, Rendezvous(dist.HashStore(), 0, 1), None)
    g = torch.Generator(device=dev).manual_seed(F)
    rand = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=dev) * std).bfloat16()
    x, dy, wr, w1, w2 = rand(T, D), rand(T, D), rand(E, D, std=0.1), rand(E, 2 * F, D, std=0.05), rand(E, D, F, std=0.05)
    moe = EPMoE(ctx, T, D, F, E, k)
    X, W1, W2, WR = (t.float().requires_grad_(True) for t in (x, w1, w2, wr))
    want = moe_reference(X, WR, W1, W2, k)
    grads = torch.autograd.grad((want * dy.float()).sum(), (X, W1, W2))
    for _ in range(5):
        out = moe.forward(x, wr, w1.view(-1, D), w2.view(-1, F))
        dx, dwr, dw1, dw2 = moe.backward(dy)
        check_status()
        # expert by expert, and the first and last rows of each by themselves
        for got, ref in ((dw1.view_as(w1), grads[1]), (dw2.view_as(w2), grads[2])):
            for e in range(E):
                for part in (slice(None), slice(0, 64), slice(-64, None)):
                    _close(got[e, part], ref[e, part], 5e-2)
        _close(dx, grads[0], 5e-2)
        _close(out, want, 3e-2)
    ctx.heap.close()
