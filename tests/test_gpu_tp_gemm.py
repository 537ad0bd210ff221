"""tcgen05 GEMM and the fused tensor-parallel kernels against PyTorch references."""
import pytest
import torch

from tests._mp import run_ranks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 256), (256, 512, 128), (1024, 3584, 1024),
                                   (2048, 1024, 8192)])
@pytest.mark.parametrize("pair", [2, 1, 0])
def test_tcgen05_gemm_matches_fp32_reference(M, N, K, pair, monkeypatch):
    """pair=2: the persistent kernel with CTA pairs (cta_group::2, 256-row tiles); 0: with single CTAs;
    1: whatever the size picks, the split kernel among it."""
    from flagcx_b200.parallel.tp import gemm_bf16
    monkeypatch.setenv("FLAGCX_GEMM_PAIR", str(pair))
    monkeypatch.setenv("FLAGCX_GEMM_SPLIT", "0" if pair == 1 else "1")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.randn(M, K, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(N, K, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    out = gemm_bf16(a, b)
    torch.cuda.synchronize()
    ref = a.float() @ b.float().T
    # bf16 output of an fp32 accumulation: half an ulp of the result, relative to its scale
    err = ((out.float() - ref).abs() / (ref.abs().mean() + ref.abs())).max().item()
    assert err < 2 ** -7, err


# parts that do not divide K's steps or the 128 rows of a tile and one step per part, with every
# tile width; and what the size rule picks (parts 0), on both sides of its lines
@pytest.mark.parametrize("M,N,K,parts,tile_n",
                         [(M, N, K, parts, t) for M, N, K, parts in
                          [(128, 256, 512, 8), (128, 512, 2112, 3), (384, 256, 576, 5), (256, 768, 1024, 7), (128, 256, 128, 2)]
                          for t in (256, 128, 64)] +
                         [(M, N, K, 0, 256) for M, N, K in
                          [(128, 256, 256), (128, 3584, 8192), (1024, 2048, 320), (512, 256, 4160), (896, 2048, 2240),
                           (1664, 768, 1024), (256, 256, 5120)]])
def test_gemm_with_k_split_over_a_cluster(M, N, K, parts, tile_n, monkeypatch):
    from flagcx_b200.parallel.tp import gemm_bf16
    monkeypatch.setenv("FLAGCX_GEMM_SPLIT", str(parts))
    monkeypatch.setenv("FLAGCX_GEMM_SPLIT_N", str(tile_n))
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    gemm_bf16(a, b, out)
    ref = a.double() @ b.double().T
    # one rounding to bf16 (2^-9 of the value) and fp32 sums of K products: each of the K additions
    # errs by at most 2^-24 of the running sum, bounded by the sum of the products' magnitudes
    bound = ref.abs() * 2 ** -8 + (a.double().abs() @ b.double().abs().T) * K * 2 ** -24
    assert bool(((out.double() - ref).abs() <= bound).all())


# full waves by the persistent kernel, the rest of the tiles by the split one: CTA pairs, single
# CTAs, and row blocks that do not fill the tile order's last group
@pytest.mark.parametrize("M,N,K,pair", [(2048, 2816, 8192, 1), (1408, 3584, 4096, 1), (2816, 1792, 4096, 1),
                                        (1408, 3584, 4096, 0), (2816, 1792, 4096, 0)])
def test_gemm_whose_last_wave_is_nearly_empty(M, N, K, pair, monkeypatch):
    from flagcx_b200.parallel.tp import gemm_bf16
    monkeypatch.setenv("FLAGCX_GEMM_PAIR", str(pair))
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    gemm_bf16(a, b, out)
    ref = a.double() @ b.double().T
    # the bound of the test above
    bound = ref.abs() * 2 ** -8 + (a.double().abs() @ b.double().abs().T) * K * 2 ** -24
    assert bool(((out.double() - ref).abs() <= bound).all())


# CTA pairs whose last row of tiles is half empty: alone, in the order's last group, over several
# waves, and with the last wave (the half tile is in it) on the split kernel.  Rows of A behind its
# end would make a sum infinite, rows of the output behind its end must stay as they are.  And what
# the size picks (pair 1): both sides for even and odd numbers of blocks.
@pytest.mark.parametrize("M,N,K,split,pair", [(128, 256, 64, 1, 2), (640, 512, 320, 1, 2), (2176, 768, 192, 1, 2),
                                              (3712, 4352, 256, 1, 2), (2176, 2816, 8192, 0, 2), (4736, 1024, 4096, 0, 2),
                                              (2304, 3072, 256, 0, 1), (2304, 3072, 1024, 0, 1),
                                              (2176, 3072, 256, 0, 1), (2176, 3072, 1024, 0, 1)])
def test_cta_pairs_with_an_odd_number_of_row_blocks(M, N, K, split, pair, monkeypatch):
    from flagcx_b200.parallel.tp import gemm_bf16
    monkeypatch.setenv("FLAGCX_GEMM_PAIR", str(pair))
    monkeypatch.setenv("FLAGCX_GEMM_SPLIT", str(split))
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    wide = torch.full((M + 128, K), float("inf"), dtype=torch.bfloat16, device="cuda")
    wide[:M] = torch.randn(M, K, generator=g, device="cuda")
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 128, N), 7.0, dtype=torch.bfloat16, device="cuda")
    a = wide[:M]
    gemm_bf16(a, b, out[:M])
    ref = a.double() @ b.double().T
    # the bound of the tests above
    bound = ref.abs() * 2 ** -8 + (a.double().abs() @ b.double().abs().T) * K * 2 ** -24
    assert bool(((out[:M].double() - ref).abs() <= bound).all())
    assert bool((out[M:] == 7).all())


# A product starts while the one in front of it ends.  Each reads what the last wrote, into buffers
# that are used again every third time: by the split kernel, the persistent one (CTA pairs and single
# CTAs), and both (full waves and a split last one); plainly and captured.
@pytest.mark.parametrize("M,N", [(128, 1024), (256, 2048), (640, 8192), (2048, 3328), (384, 8192)])
def test_products_that_follow_one_another(M, N):
    from flagcx_b200.parallel.tp import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, N, generator=g, device="cuda") * N ** -0.5).to(torch.bfloat16)

    def chain(wait):
        bufs = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3)]
        src = x
        for i in range(7):
            gemm_bf16(src, w, bufs[i % 3])
            if wait:
                torch.cuda.synchronize()
            src = bufs[i % 3]
        return src

    want = chain(True)
    assert bool(torch.isfinite(want).all())
    for _ in range(3):
        assert torch.equal(chain(False), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(False)
    for _ in range(3):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs at least 2 GPUs")
def test_fused_tensor_parallel_kernels_on_real_peers():
    n = 8 if torch.cuda.device_count() >= 8 else 4 if torch.cuda.device_count() >= 4 else 2
    res = run_ranks(n, "tp_fused", 128 * n * 2, 512, 1024, timeout=300)
    for rank, errs in res.items():
        assert errs["ag_gemm"] < 2 ** -6 and errs["gemm_rs"] < 2 ** -5, (rank, errs)
