"""Fused model kernels and the sharding engine against plain PyTorch fp32 references."""
import pytest
import torch
import torch.nn.functional as F

from tests._mp import run_ranks

pytestmark = pytest.mark.gpu


def _ops():
    from flagcx_b200 import ops
    ops.ext()  # must be the compiled extension
    return ops


def test_rmsnorm_forward_backward():
    ops = _ops()
    torch.manual_seed(0)
    # widths: each forward variant (4 / 8 / 16 packs per lane, then one CTA per row); the backward
    # in groups with several rows each (2500, 700 rows) and with one row per CTA, most of the grid
    # without work (37 rows)
    for rows, H in ((2500, 256), (37, 1000), (37, 2048), (2500, 4096), (37, 4096), (700, 8192), (37, 16384)):
        x = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        w = (1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16).requires_grad_()
        y = ops.rmsnorm(x, w, 1e-5)
        g = torch.randn_like(y)
        y.backward(g)
        xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
        yr = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
        yr.backward(g.float())
        assert (y.float() - yr).abs().max() < 0.05
        assert (x.grad.float() - xf.grad).abs().max() < 0.05
        assert ((w.grad.float() - wf.grad).abs() / wf.grad.abs().clamp(min=1)).max() < 0.05, (rows, H)


# one row per CTA (one and two packs of 8 per thread) and two, to the last count of rows; then every
# group size (32 to 512 threads, one to four packs each), from the first count of rows that takes
# groups to several more rows than a ring has slots, which the groups share unevenly
@pytest.mark.parametrize("rows,H", [(1, 8), (17, 256), (5, 1024), (33, 1032), (300, 2048), (7, 2056), (149, 3688), (149, 3680),
                                    (9, 4104), (200, 7176), (3, 8200), (5, 12296), (2, 16384), (2500, 264),
                                    (148, 8192), (592, 1024), (593, 1024), (444, 3584), (445, 4096), (296, 2560), (297, 2560),
                                    (17000, 256), (16600, 1024), (4800, 2048), (9000, 1288), (4200, 2560), (2500, 4096),
                                    (1300, 7176), (2000, 5120), (1300, 8192), (1000, 12296), (700, 16384)])
@pytest.mark.parametrize("skip", [True, False])
def test_rmsnorm_backward_at_the_edges_of_its_row_groups(rows, H, skip):
    ops = _ops()
    gen = torch.Generator(device="cuda").manual_seed(rows + H)
    x, g, gs = [torch.randn(rows, H, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(3)]
    w = (1 + 0.1 * torch.randn(H, generator=gen, device="cuda")).to(torch.bfloat16)
    x.requires_grad_()
    w.requires_grad_()
    if skip:
        dx, dw = torch.autograd.grad(ops.rmsnorm_branch(x, w, 1e-5), (x, w), (g, gs))
    else:
        dx, dw = torch.autograd.grad(ops.rmsnorm(x, w, 1e-5), (x, w), g)
    xd, wd, gd = x.detach().double().requires_grad_(), w.detach().double().requires_grad_(), g.double()
    xhat = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)
    rdx, rdw = torch.autograd.grad(xhat * wd, (xd, wd), gd)
    if skip:
        rdx = rdx + gs.double()
    # one rounding to bf16; the fp32 terms before it are a few and at most |g w| + |x| + |skip| large
    scale = (gd * wd).abs() + xd.abs() + gs.double().abs()
    assert bool(((dx.double() - rdx).abs() <= rdx.abs() * 2 ** -8 + scale.detach() * 2 ** -18).all())
    terms = (gd * xhat).abs().sum(0).detach()
    assert bool(((dw.double() - rdw).abs() <= rdw.abs() * 2 ** -8 + terms * 2 ** -16).all())


# one row per warp up to 256 threads per row, the ends of each (a pack less, a pack more), CTAs whose
# last rows do not exist, and eight packs per thread
@pytest.mark.parametrize("H", [8, 256, 264, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("rows", [1, 3, 4, 301])
def test_norm_forward_at_the_edges_of_its_groups(H, rows):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(H + rows)
    x = torch.randn(rows, H, generator=g, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16)
    y, rstd = ops.ext().rmsnorm_fwd(x, w, 1e-5)
    want = torch.rsqrt(x.double().square().mean(-1) + 1e-5)
    # fp32 sums of H squares, then rsqrtf: a few units in the last place of H additions at most
    assert bool(((rstd.double() - want).abs() <= want * (H + 8) * 2 ** -24).all())
    ref = x.double() * want[:, None] * w.double()
    assert bool(((y.double() - ref).abs() <= ref.abs() * (2 ** -8 + (H + 16) * 2 ** -24)).all())  # and one rounding to bf16
    x[0, H // 2] = float("inf")  # the row's sum: 0 for what is finite, NaN for the infinity
    y2, _ = ops.ext().rmsnorm_fwd(x, w, 1e-5)
    assert bool(y2[0, H // 2].isnan()) and int(y2[0].isnan().sum()) == 1 and torch.equal(y2[1:], y[1:])


def test_norm_backward_from_two_threads_with_different_sizes():
    """The backward of an autograd graph runs without the GIL, so its launches interleave with
    another thread's; 8 and 256 columns share a kernel and ask for 3 and 144 KiB of shared memory."""
    import threading
    import time
    ops = _ops()
    made = {}
    for H in (8, 256):
        x, g, skip = [torch.randn(300, H, device="cuda").to(torch.bfloat16) for _ in range(3)]
        w = torch.ones(H, device="cuda", dtype=torch.bfloat16)
        made[H] = x, w, g, skip, ops.ext().rmsnorm_fwd(x, w, 1e-5)[1]
    errors, stop = [], threading.Event()

    def small():
        x, w, g, _, rstd = made[8]
        try:
            while not stop.is_set():
                for _ in range(20):
                    ops.ext().rmsnorm_bwd(g, x, w, rstd)
                torch.cuda.synchronize()  # a full launch queue would keep the other thread out
        except RuntimeError as e:
            errors.append(e)

    other = threading.Thread(target=small)
    other.start()
    try:
        x, w, g, skip, _ = made[256]
        x.requires_grad_()
        end = time.monotonic() + 3
        while time.monotonic() < end:
            torch.autograd.grad(ops.rmsnorm_branch(x, w, 1e-5), x, (g, skip))
    finally:
        stop.set()
        other.join()
    torch.cuda.synchronize()
    assert not errors, errors


def test_operators_keep_hooks_tracing_and_transforms():
    """The operators run as C++ autograd functions, except under a tracer, a function transform or
    forward-mode differentiation."""
    ops = _ops()
    x = torch.randn(5, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    w, g = torch.ones_like(x[0]).requires_grad_(), torch.randn_like(x)
    before = ops.launch_count
    plain = torch.autograd.grad(ops.rmsnorm(x, w), (x, w), g)
    assert ops.launch_count - before == 2
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (saved.append(1), t.cpu())[1], lambda t: t.cuda()):
        y = ops.rmsnorm(x, w)
    assert len(saved) == 3 and all(torch.equal(a, b) for a, b in zip(plain, torch.autograd.grad(y, (x, w), g)))
    other = torch.randn_like(g)
    traced = torch.jit.trace(lambda t: ops.swiglu(t), (g,), check_trace=False)
    assert torch.equal(traced(other), ops.swiglu(other))
    with pytest.raises(RuntimeError, match="functorch transforms"):
        torch.vmap(ops.swiglu)(g[None])
    with torch.autograd.forward_ad.dual_level(), pytest.raises(NotImplementedError):
        ops.swiglu(torch.autograd.forward_ad.make_dual(g, other))
    own = type("Own", (torch.Tensor,), {})
    y, skip = ops.rmsnorm_branch(g.as_subclass(own), w)
    assert type(skip) is own and torch.equal(y, ops.rmsnorm(g, w))


def test_results_without_memory_are_refused():
    """Under a mode that makes every new tensor a fake one."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    ops = _ops()
    x = torch.randn(3, 512, device="cuda").to(torch.bfloat16)
    for call in (lambda: ops.swiglu(x), lambda: ops.rmsnorm(x, x[0]), lambda: ops.rope_fused_qkv(x, 4, 2, 64),
                 lambda: ops.ext().swiglu_bwd(x, torch.cat([x, x], 1))):
        with FakeTensorMode(allow_non_fake_inputs=True), pytest.raises(RuntimeError, match="not allocated"):
            call()
    assert not ops.swiglu(x).isnan().any()


def test_rope_matches_reference_and_backward_is_inverse():
    ops = _ops()
    T, Hn, D = 64, 4, 128
    x = torch.randn(T, Hn, D, device="cuda", dtype=torch.bfloat16)
    y = ops.rope(x, 500000.0)
    half = D // 2
    inv = 500000.0 ** (-torch.arange(0, half, device="cuda", dtype=torch.float32) * 2 / D)
    ang = torch.arange(T, device="cuda", dtype=torch.float32)[:, None] * inv[None]
    c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
    x1, x2 = x[..., :half].float(), x[..., half:].float()
    ref = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)
    assert (y.float() - ref).abs().max() < 0.03
    xg = x.clone().requires_grad_()
    ops.rope(xg, 500000.0).backward(y)  # rotating back a rotated vector gives the original
    assert (xg.grad.float() - x.float()).abs().max() < 0.06


def test_rope_on_the_fused_projection_rotates_q_and_k_and_copies_v():
    ops = _ops()
    T, nh, nkv, D = 70, 8, 2, 128
    qkv = torch.randn(T, (nh + 2 * nkv) * D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    out = ops.rope_fused_qkv(qkv, nh, nkv, D, 500000.0)
    q, k, v = out.split([nh * D, nkv * D, nkv * D], dim=-1)
    q0, k0, v0 = qkv.detach().split([nh * D, nkv * D, nkv * D], dim=-1)
    assert torch.equal(v, v0)
    half = D // 2
    inv = 500000.0 ** (-torch.arange(0, half, device="cuda", dtype=torch.float32) * 2 / D)
    ang = torch.arange(T, device="cuda", dtype=torch.float32)[:, None] * inv[None]
    c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def rot(x, heads):
        x = x.reshape(T, heads, D).float()
        x1, x2 = x[..., :half], x[..., half:]
        return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).reshape(T, heads * D)

    assert (q.float() - rot(q0, nh)).abs().max() < 0.03
    assert (k.float() - rot(k0, nkv)).abs().max() < 0.03
    # backward: the rotation's transpose on q and k (rotating back what was rotated), identity on v
    out.backward(out.detach())
    gq, gk, gv = qkv.grad.split([nh * D, nkv * D, nkv * D], dim=-1)
    assert (gq.float() - q0.float()).abs().max() < 0.06
    assert (gk.float() - k0.float()).abs().max() < 0.06
    assert torch.equal(gv, v0)


def test_norm_branch_and_residual_linear_match_the_unfused_graph():
    """y = linear(f(norm(x)), w) + x, written with rmsnorm_branch / linear(residual=...),
    against the same expression in fp32: output, dx (skip gradient added inside the norm's
    backward), dw of the norm and of the linear."""
    ops = _ops()
    torch.manual_seed(1)
    T, H = 333, 1024
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    wn = (1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16).requires_grad_()
    w = (0.03 * torch.randn(H, H, device="cuda")).to(torch.bfloat16).requires_grad_()
    h, skip = ops.rmsnorm_branch(x, wn, 1e-5)
    y = ops.linear(h, w, residual=skip)
    g = torch.randn_like(y)
    y.backward(g)
    xf, wnf, wf = (t.detach().float().requires_grad_() for t in (x, wn, w))
    hf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wnf
    yf = hf @ wf.T + xf
    yf.backward(g.float())
    assert (y.float() - yf).abs().max() < 0.06
    assert (x.grad.float() - xf.grad).abs().max() < 0.06
    # the weight gradients are sums over 333 rows of bf16 products: compare in the L2 norm
    assert (wn.grad.float() - wnf.grad).norm() / wnf.grad.norm() < 0.01
    assert (w.grad.float() - wf.grad).norm() / wf.grad.norm() < 0.01
    # only the skip connection used: the gradient passes through untouched
    x2 = x.detach().clone().requires_grad_()
    _, skip2 = ops.rmsnorm_branch(x2, wn.detach(), 1e-5)
    skip2.backward(g)
    assert torch.equal(x2.grad, g)
    # one output used, in both implementations: the other one's gradient counts as zeros
    for fn in (ops.rmsnorm_branch, ops._RMSNormBranch.apply):
        dx, dw = torch.autograd.grad(fn(x, wn, 1e-5)[1], (x, wn), g)
        assert torch.equal(dx, g) and not dw.any()
        one = torch.autograd.grad(fn(x, wn, 1e-5)[0], (x, wn), g)
        assert all(torch.equal(a, b) for a, b in zip(one, torch.autograd.grad(ops.rmsnorm(x, wn, 1e-5), (x, wn), g)))


def test_swiglu_forward_backward():
    ops = _ops()
    ab = torch.randn(50, 2 * 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    out = ops.swiglu(ab)
    g = torch.randn_like(out)
    out.backward(g)
    abf = ab.detach().float().requires_grad_()
    ref = F.silu(abf[:, :512]) * abf[:, 512:]
    ref.backward(g.float())
    assert (out.float() - ref).abs().max() < 0.05
    assert (ab.grad.float() - abf.grad).abs().max() < 0.06


# vocabulary sizes: one CTA per row; the Llama-3 vocabulary (a cluster of 4 CTAs per row);
# a row that does not divide evenly over its cluster; parts above 72 KiB (one CTA per SM);
# a row too long for shared memory (the kernel that streams it three times)
@pytest.mark.parametrize("T,V", [(33, 1024), (9, 128256), (5, 50264), (3, 300000), (2, 2000000)])
def test_cross_entropy_loss_and_gradient(T, V):
    ops = _ops()
    logits = (3 * torch.randn(T, V, device="cuda")).to(torch.bfloat16)
    tgt = torch.randint(0, V, (T,), device="cuda")
    lf = logits.float().requires_grad_()
    ref = F.cross_entropy(lf, tgt)
    ref.backward()
    work = logits.clone().requires_grad_()
    w2 = work * 1.0  # non-leaf, as in the model (the kernel overwrites it)
    loss = ops.cross_entropy_(w2, tgt)
    loss.backward()
    assert abs(float(loss) - float(ref)) < 2e-3
    assert (work.grad.float() - lf.grad).abs().max() < 2e-3
    # relative check where the gradient is not tiny: two bf16 roundings at most
    big = lf.grad.abs() > 1e-4
    if big.any():
        rel = ((work.grad.float() - lf.grad).abs() / lf.grad.abs())[big].max()
        assert rel < 1.2e-2


# few rows, which are spread over up to eight CTAs each; then the edges of what one CTA holds (256
# threads x 1, 2, 4, 8, 10, 13, 16 packs of 8) with 300 rows and more, so that a row stays with as few
# CTAs as can hold it, and with several rows for each of them: one (up to 32768 columns), two, four
# and eight CTAs per row; the last row size of the persistent kernel and the first of the next one.
# A stretch of -inf (masked vocabulary) in every second row
@pytest.mark.parametrize("T,V", [(1, 8), (3, 2048), (5, 2056), (2, 4104), (3, 8200), (2, 16392), (2, 20488), (3, 32768),
                                 (2, 32776), (7, 65544), (2, 151936), (700, 128256), (2, 262144), (2, 262152),
                                 (5000, 1024), (3000, 2048), (3000, 2056), (3000, 4096), (3000, 4104), (1500, 8192), (1500, 8200),
                                 (900, 16384), (700, 16392), (700, 20480), (500, 20488), (500, 26624), (500, 26632), (500, 32768),
                                 (500, 32776), (400, 40960), (400, 65536), (300, 65544), (300, 100352), (300, 131080),
                                 (300, 151936), (300, 262144)])
def test_cross_entropy_at_the_edges_of_its_row_split(T, V):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = (torch.randn(T, V, generator=g, device="cuda") * 3).to(torch.bfloat16)
    tgt = torch.randint(0, V // 2, (T,), generator=g, device="cuda")
    tgt[0] = V - 1
    logits[1::2, V // 2:] = float("-inf")
    lp = logits.double().log_softmax(-1)
    at = torch.arange(T, device="cuda")
    want = -lp[at, tgt].mean()
    d = lp.exp_()
    d[at, tgt] -= 1
    d /= T
    loss = ops.cross_entropy_(logits, tgt)
    assert abs(loss.double() - want) <= 1e-5 * want + 1e-5
    # the exponential and the gradient are each rounded to bf16 (2^-9 of the value each), the
    # fp32 exponential and the sum add less than 2^-15; at the target softmax and 1 cancel
    assert bool(((logits.double() - d).abs() <= d.abs() * 2 ** -7 + 2 ** -15 / T * (d < 0)).all())


# Rows dealt out: the edges of what one CTA holds (256 threads x 4, 8, 10, 13, 16, 18, 21 packs of 8) with
# as few rows as are dealt, and one, two, three, five and seven CTAs per row.  Two rows hold a NaN: they
# are lost, and their clusters take over no others, which are done all the same.
@pytest.mark.parametrize("T,V", [(5925, 4104), (5920, 8192), (4737, 8200), (4736, 16384), (3555, 16392), (3552, 20480), (2370, 20488),
                                 (2368, 26624), (2368, 26632), (2369, 32768), (2368, 32776), (2368, 36864), (2368, 36872),
                                 (2371, 43008), (1184, 43016), (790, 86024), (475, 172040), (340, 262144)])
def test_cross_entropy_of_rows_dealt_out(T, V):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = (torch.randn(T, V, generator=g, device="cuda") * 3).to(torch.bfloat16)
    tgt = torch.randint(0, V // 2, (T,), generator=g, device="cuda")
    tgt[0] = V - 1
    logits[1::2, V // 2:] = float("-inf")
    bad = [3, T // 2]
    logits[bad, 1] = float("nan")
    lp = logits.double().log_softmax(-1)
    at = torch.arange(T, device="cuda")
    want = -lp[at, tgt]
    d = lp.exp_()
    d[at, tgt] -= 1
    loss = ops.ext().cross_entropy_fwd_bwd_(logits, tgt, 1.0)
    good = torch.ones(T, dtype=torch.bool, device="cuda")
    good[bad] = False
    assert bool(loss[~good].isnan().all()) and bool(logits[~good].isnan().any(1).all())
    assert bool(((loss.double() - want).abs()[good] <= 1e-5 * want[good].abs() + 1e-5).all())
    # bounds of the test above, for a scale of 1
    assert bool(((logits.double() - d).abs() <= d.abs() * 2 ** -7 + 2 ** -15 * (d < 0))[good].all())


def test_adamw_matches_torch():
    ops = _ops()
    torch.manual_seed(5)
    n = 10007
    p = torch.randn(n, device="cuda").to(torch.bfloat16)
    g = torch.randn(n, device="cuda").to(torch.bfloat16)
    m = torch.zeros_like(p)
    v = torch.zeros_like(p)
    pr = torch.nn.Parameter(p.float().clone())
    opt = torch.optim.AdamW([pr], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in (1, 2, 3):
        pr.grad = g.float()
        opt.step()
        ops.adamw_flat_(p, g, m, v, 1e-2, 0.9, 0.95, 1e-8, 0.1, step)
    # parameters and both moments are rounded to bf16 after every step: half an ulp each time,
    # i.e. 2^-9 relative for |p| >= 1 and 2^-9 absolute below
    assert ((p.float() - pr.detach()).abs() / pr.detach().abs().clamp(min=1)).max() < 0.02


def test_sharded_engine_world1_matches_fp32_reference():
    from flagcx_b200 import ops
    from flagcx_b200.models.llama import LlamaConfig, build_units, reference_forward
    from flagcx_b200.parallel.fsdp import ShardedModel
    cfg = LlamaConfig.tiny()
    ops.assume_unit_loss_grad = True
    model = ShardedModel(build_units(cfg), None, 0, 1, torch.device("cuda", 0), lr=1e-3)
    tok = torch.randint(0, cfg.vocab, (129,), device="cuda")
    params = model.full_parameters()
    ref = reference_forward(cfg, params, tok[:-1], tok[1:])
    loss0 = model.train_step(tok[:-1], tok[1:])
    assert abs(float(loss0) - float(ref)) < 0.05, (float(loss0), float(ref))
    losses = [float(model.train_step(tok[:-1], tok[1:])) for _ in range(8)]
    assert losses[-1] < float(loss0) - 0.5, (float(loss0), losses)  # it learns the batch
    model.close()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs at least 2 GPUs")
def test_sharded_engine_world2_matches_world1():
    """Same seed, same batch on every rank: the sharded run must reproduce the
    single-GPU losses (gradients are averaged over identical replicas)."""
    from tests.test_cpu_torch_backend import free_port
    one = run_ranks(1, "fsdp_losses", free_port(), 4, timeout=300)[0]
    two = run_ranks(2, "fsdp_losses", free_port(), 4, timeout=300)
    for a, b in zip(one, two[0]):
        assert abs(a - b) < 0.05, (one, two[0])
    assert two[0] == two[1]


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs at least 2 GPUs")
def test_torch_fsdp_over_flagcx_matches_nccl():
    """torch.distributed.fsdp.fully_shard with backend='flagcx' trains like backend='nccl'."""
    from tests.test_cpu_torch_backend import free_port
    ours = run_ranks(2, "torch_fsdp2_losses", free_port(), "flagcx", timeout=300)
    nccl = run_ranks(2, "torch_fsdp2_losses", free_port(), "nccl", timeout=300)
    for a, b in zip(ours[0], nccl[0]):
        assert abs(a - b) <= 0.02 * max(1.0, abs(b)), (ours[0], nccl[0])


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs at least 2 GPUs")
def test_torch_backend_ops_on_gpus():
    from tests.test_cpu_torch_backend import free_port
    n = 2
    res = run_ranks(n, "torch_backend_ops", free_port(), True, timeout=300)
    assert all(v == "ok" for v in res.values())


def test_optimizer_under_backward_gives_the_same_model():
    """AdamW of a unit queued right behind that unit's gradients (on its own stream, under
    the rest of the backward pass) against AdamW after the whole backward pass: same
    losses, same parameters."""
    from flagcx_b200 import ops
    from flagcx_b200.models.llama import LlamaConfig, build_units
    from flagcx_b200.parallel.fsdp import ShardedModel
    cfg = LlamaConfig.tiny()
    ops.assume_unit_loss_grad = True
    g = torch.Generator().manual_seed(3)
    batches = [torch.randint(0, cfg.vocab, (129,), generator=g).cuda() for _ in range(4)]
    runs = []
    for overlap in (False, True):
        m = ShardedModel(build_units(cfg), None, 0, 1, torch.device("cuda", 0), overlap_optimizer=overlap)
        losses = [float(m.train_step(b[:-1], b[1:])) for b in batches]
        torch.cuda.synchronize()
        runs.append((losses, [s.clone() for s in m.shard]))
        m.close()
    (la, pa), (lb, pb) = runs
    assert max(abs(x - y) for x, y in zip(la, lb)) < 2e-2, (la, lb)
    for x, y in zip(pa, pb):
        assert (x.float() - y.float()).abs().max().item() < 2e-2


def test_checkpoint_round_trip_resumes_with_the_same_loss():
    """state_dict -> load_state_dict into a fresh engine: the next step's loss is the one
    the original engine computes (parameters, both AdamW moments and the step counter)."""
    from flagcx_b200 import ops
    from flagcx_b200.models.llama import LlamaConfig, build_units
    from flagcx_b200.parallel.fsdp import ShardedModel
    cfg = LlamaConfig.tiny()
    ops.assume_unit_loss_grad = True
    g = torch.Generator().manual_seed(11)
    batches = [torch.randint(0, cfg.vocab, (129,), generator=g).cuda() for _ in range(4)]
    a = ShardedModel(build_units(cfg), None, 0, 1, torch.device("cuda", 0), lr=1e-3)
    for b in batches[:2]:
        a.train_step(b[:-1], b[1:])
    sd = a.state_dict()
    want = [float(a.train_step(b[:-1], b[1:])) for b in batches[2:]]
    fresh = ShardedModel(build_units(cfg), None, 0, 1, torch.device("cuda", 0), lr=1e-3, seed=999)  # other weights
    fresh.load_state_dict(sd)
    got = [float(fresh.train_step(b[:-1], b[1:])) for b in batches[2:]]
    assert fresh.step_count == a.step_count
    assert max(abs(x - y) for x, y in zip(want, got)) < 2e-2, (want, got)
    a.close()
    fresh.close()
