"""What the model kernels and the GEMM that splits K make of a copy that never comes, or too late: the
wait for it runs out (20 ms in this build of them), the kernel ends, what depends on it is NaN and
everything else is right."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from flagcx_b200.build import build_opwait
    torch.cuda.init()
    so = ctypes.CDLL(build_opwait())
    so.hold_back.argtypes = [ctypes.c_long]
    so.norm_forward.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_long, ctypes.c_int]
    so.norm_partials.argtypes = [ctypes.c_long, ctypes.c_int, ctypes.c_int]
    so.norm_backward.argtypes = [ctypes.c_void_p] * 8 + [ctypes.c_long, ctypes.c_int, ctypes.c_int]
    so.cross_entropy.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_long, ctypes.c_int, ctypes.c_float, ctypes.c_int]
    yield so
    so.hold_back(-1)
    so.leave_unseen(0, 0, 0)


# the longest rows of every group of threads, and rows that no kernel holds
@pytest.mark.parametrize("H,held", [(1024, 1), (2048, 1), (4096, 1), (8192, 1), (8200, 1), (16384, 1), (16392, 0), (32768, 0)])
def test_norm_forward_takes_rows_that_a_kernel_holds_and_no_others(lib, H, held):
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(5, H, generator=g, device="cuda").to(torch.bfloat16)
    w, y, rstd = torch.ones_like(x[0]), torch.full_like(x, 7.0), torch.full((5,), 7.0, device="cuda")
    assert (lib.norm_forward(*[t.data_ptr() for t in (x, w, y, rstd)], 5, H) == 0) == bool(held)
    ref = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) if held else torch.full_like(x, 7.0).double()
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2 ** -8).all())  # one rounding to bf16, and fp32 in front of it


def _norm_backward(lib, t, rows, H, skip, held):
    assert lib.hold_back(held) == 0
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    dx, dw = torch.full_like(t["x"], 7.0), torch.full_like(t["w"], 7.0)
    partial = torch.empty(lib.norm_partials(rows, H, sms), H, device="cuda")
    assert lib.norm_backward(*[p.data_ptr() for p in (t["g"], t["x"], t["w"], t["rstd"])], t["skip"].data_ptr() if skip else None,
                             dx.data_ptr(), dw.data_ptr(), partial.data_ptr(), rows, H, sms) == 0
    return dx, dw


# groups of 32 to 512 threads with rows for several rounds of their rings, and few rows: one per
# CTA (with one and two packs per thread) or two
@pytest.mark.parametrize("rows,H,skip", [(9000, 256, 1), (4000, 1032, 0), (3000, 2560, 1), (2000, 5120, 0), (700, 12296, 1),
                                         (5000, 4096, 1), (100, 4096, 1), (148, 8192, 0), (592, 2048, 0), (500, 1024, 1)])
def test_norm_backward_without_one_row(lib, rows, H, skip):
    g = torch.Generator(device="cuda").manual_seed(rows)
    t = {k: torch.randn(rows, H, generator=g, device="cuda").to(torch.bfloat16) for k in ("x", "g", "skip")}
    t["w"] = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    t["rstd"] = torch.rsqrt(t["x"].float().square().mean(-1) + 1e-5)
    whole = _norm_backward(lib, t, rows, H, skip, -1)
    assert not whole[0].isnan().any() and not whole[1].isnan().any()
    held = rows // 2 + 1
    dx, dw = _norm_backward(lib, t, rows, H, skip, held)
    lost = dx.isnan().any(1)
    assert torch.equal(lost, dx.isnan().all(1)) and bool(lost[held])  # a row is lost as a whole
    assert 0 < int(lost.sum()) <= rows - held and not bool(lost[:held].any())  # from there on, in one group
    assert torch.equal(dx[~lost], whole[0][~lost])
    assert bool(dw.isnan().all())
    again = _norm_backward(lib, t, rows, H, skip, -1)
    assert all(torch.equal(a, b) for a, b in zip(again, whole))


def _cross_entropy(lib, logits, targets, held):
    assert lib.hold_back(held) == 0
    rows, V = logits.shape
    d, loss = logits.clone(), torch.full((rows,), 7.0, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lib.cross_entropy(d.data_ptr(), targets.data_ptr(), loss.data_ptr(), rows, V, 1.0 / rows, sms) == 0
    return d, loss


# one, two, four and eight CTAs per row, with several rows for each, and the kernel that takes one
# row per cluster
@pytest.mark.parametrize("rows,V", [(5000, 1024), (900, 32768), (700, 65536), (600, 128256), (300, 262144), (5, 262152)])
def test_cross_entropy_without_one_row(lib, rows, V):
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(rows, V, generator=g, device="cuda").to(torch.bfloat16)
    targets = torch.randint(0, V, (rows,), generator=g, device="cuda")
    whole = _cross_entropy(lib, logits, targets, -1)
    assert not whole[0].isnan().any() and not whole[1].isnan().any()
    held = rows // 2 + 1
    d, loss = _cross_entropy(lib, logits, targets, held)
    lost = loss.isnan()
    assert bool(lost[held]) and not bool(lost[:held].any()) and not bool(lost[held:].all())
    assert bool(d[lost].isnan().all())
    assert torch.equal(loss[~lost], whole[1][~lost]) and torch.equal(d[~lost], whole[0][~lost])
    again = _cross_entropy(lib, logits, targets, -1)
    assert all(torch.equal(a, b) for a, b in zip(again, whole))


# rows dealt out to the clusters: the one that lost a copy had the next two rows already, and takes no more
@pytest.mark.parametrize("rows,V", [(8000, 8192), (2400, 43008), (1000, 128256), (400, 262144)])
def test_cross_entropy_of_rows_dealt_out_without_one(lib, rows, V):
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(rows, V, generator=g, device="cuda").to(torch.bfloat16)
    targets = torch.randint(0, V, (rows,), generator=g, device="cuda")
    whole = _cross_entropy(lib, logits, targets, -1)
    held = rows // 2 + 1
    d, loss = _cross_entropy(lib, logits, targets, held)
    lost = loss.isnan()
    assert bool(lost[held]) and not bool(lost[:held].any()) and int(lost.sum()) <= 3
    assert bool(d[lost].isnan().all())
    assert torch.equal(loss[~lost], whole[1][~lost]) and torch.equal(d[~lost], whole[0][~lost])


# The answer to a cluster's first request, or a later one, is not seen in time.  Seen while the cluster
# waits once more, the row that it hands over is done like any other; not seen at all, that row is left
# as it was, and the cluster's own rows tell.
@pytest.mark.parametrize("rows,V,ctas", [(8000, 8192, 1), (1000, 128256, 3)])
@pytest.mark.parametrize("nth", [0, 1, 2])
def test_cross_entropy_of_rows_dealt_out_without_an_answer(lib, rows, V, ctas, nth):
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(rows, V, generator=g, device="cuda").to(torch.bfloat16)
    targets = torch.randint(0, V, (rows,), generator=g, device="cuda")
    whole = _cross_entropy(lib, logits, targets, -1)
    try:
        assert lib.leave_unseen(5 * ctas, nth, 1) == 0
        late = _cross_entropy(lib, logits, targets, -1)
        assert all(torch.equal(a, b) for a, b in zip(late, whole))
        assert lib.leave_unseen(5 * ctas, nth, 2) == 0
        d, loss = _cross_entropy(lib, logits, targets, -1)
    finally:
        lib.leave_unseen(0, 0, 0)
    lost, undone = loss.isnan(), loss == 7.0
    assert 1 <= int(lost.sum()) <= 2 and bool(d[lost].isnan().all())
    assert int(undone.sum()) == 1 and torch.equal(d[undone], logits[undone])
    rest = ~(lost | undone)
    assert torch.equal(loss[rest], whole[1][rest]) and torch.equal(d[rest], whole[0][rest])


@pytest.fixture(scope="module")
def gemm():
    from flagcx_b200.build import build_gemmwait
    torch.cuda.init()
    so = ctypes.CDLL(build_gemmwait())
    so.split_gemm.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 5
    yield so
    so.hold_back_step(-1, -1)


# A step of the first, a middle and the last part, which arrives when its CTA has given up: the whole
# ring is asked for by then (parts of 2 steps, fewer than there are stages) or the producer still waits
# for a stage (parts of 21).
@pytest.mark.parametrize("K,parts", [(1024, 8), (512, 3), (1344, 1), (5376, 4)])
@pytest.mark.parametrize("tile_n", [256, 128, 64])
def test_split_gemm_of_operands_that_come_too_late(gemm, K, parts, tile_n):
    M, N, steps = 256, 512, K // 64
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)

    def run(tile, kb):
        assert gemm.hold_back_step(tile, kb) == 0
        out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
        assert gemm.split_gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, parts, tile_n) == 0
        return out

    whole = run(-1, -1)
    ref = a.double() @ b.double().T
    # one rounding to bf16 and fp32 sums of K products
    bound = ref.abs() * 2 ** -8 + (a.double().abs() @ b.double().abs().T) * K * 2 ** -24
    assert bool(((whole.double() - ref).abs() <= bound).all())
    tile = 3 if N // tile_n > 1 else 1
    down, across = tile % (M // 128), tile // (M // 128)  # neighbours share their rows of B
    lost = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    lost[down * 128:(down + 1) * 128, across * tile_n:(across + 1) * tile_n] = True
    for kb in (0, steps // 2, steps - 1):
        out = run(tile, kb)
        assert torch.equal(out.isnan(), lost), kb
        assert torch.equal(out[~lost], whole[~lost]), kb
    assert torch.equal(run(-1, -1), whole)
