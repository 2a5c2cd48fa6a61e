"""tcgen05 GEMM kernels against an fp32 PyTorch matmul of the same bf16 inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, ref, k):
    # bf16 output of an fp32 accumulation: relative 2^-7 of the result magnitude plus a
    # small absolute term for cancellation
    err = (out.float() - ref).abs()
    tol = ref.abs() * 2 ** -7 + 2 ** -7 * ref.abs().mean() + 1e-3
    bad = (err > tol).sum().item()
    assert bad == 0, f"{bad} of {out.numel()} elements off; max err {err.max().item():.4g}"


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 4096), (1000, 4096, 4096), (77, 96, 136),
                                   (8192, 3584, 512), (4096, 1152, 256), (300, 4128, 192)])  # tile widths 224 and 192, ragged last tile
def test_gemm_bf16(m, n, k):
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = gemm.gemm_bf16(a, b, pair=False)
    torch.cuda.synchronize()
    default_status().check()
    ref = a.float() @ b.float().t()
    _check(out, ref, k)


@pytest.mark.parametrize("pair", [False, True, "wide", "swap"])
def test_grouped_gemm_store_and_swiglu(pair):
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(5)
    sizes = [0, 5, 128, 131, 300, 1, 0, 64] + ([256, 700, 513] if pair else [])
    g, k, n = len(sizes), 512, 256
    offs = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total = sum(sizes)
    a = torch.randn(total + 50, k, device="cuda", dtype=torch.bfloat16)  # extra rows past the last group are ignored
    w = (torch.randn(g, n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((total + 50, n), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_bf16(a, w, offs, out=out, pair=pair)
    torch.cuda.synchronize()
    default_status().check()
    start = 0
    for gi, sz in enumerate(sizes):
        if sz:
            ref = a[start:start + sz].float() @ w[gi].float().t()
            _check(out[start:start + sz], ref, k)
        start += sz
    assert (out[total:] == 7.0).all(), "rows outside every group must not be written"

    # SwiGLU: weights hold N gate rows then N up rows per group
    n_int = 128
    w2 = (torch.randn(g, 2 * n_int, k, device="cuda") * 0.05).to(torch.bfloat16)
    h = gemm.grouped_gemm_bf16(a, w2, offs, epilogue=gemm.EPI_SWIGLU, pair=pair)
    torch.cuda.synchronize()
    default_status().check()
    start = 0
    for gi, sz in enumerate(sizes):
        if sz:
            x = a[start:start + sz].float()
            gate = x @ w2[gi, :n_int].float().t()
            up = x @ w2[gi, n_int:].float().t()
            _check(h[start:start + sz], torch.nn.functional.silu(gate) * up, k)
        start += sz


@pytest.mark.parametrize("tile_n,w_prefetch,tile_m", [(128, 0, 0), (192, 3, 0), (224, 0, 0), (0, 4, 0), (0, 40, 0), (0, 0, 64)])
def test_grouped_gemm_narrow_tiles(tile_n, w_prefetch, tile_m):
    """The single-CTA grouped GEMM with tile widths other than 256, with the weight prefetch into L2 (a distance
    shorter and longer than the K loop of 6 blocks) and with row tiles of 64: store, SwiGLU (an output width that the
    half tile does not divide) and scatter epilogues against the fp32 product."""
    import ctypes

    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(tile_n + w_prefetch + tile_m)
    sizes = [3, 0, 130, 257, 64]
    g, k, n = len(sizes), 384, 448
    total = sum(sizes)
    offs = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    a = torch.randn(total, k, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(g, n, k, device="cuda") * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(g, 2 * n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = gemm.grouped_gemm_bf16(a, w, offs, tile_n=tile_n, w_prefetch=w_prefetch, tile_m=tile_m)
    h = gemm.grouped_gemm_bf16(a, w2, offs, epilogue=gemm.EPI_SWIGLU, tile_n=tile_n, w_prefetch=w_prefetch, tile_m=tile_m)
    dst = torch.zeros(total, n, device="cuda", dtype=torch.bfloat16)
    perm = torch.randperm(total, device="cuda")
    bases = (ctypes.c_ulonglong * 8)()
    bases[0] = dst.data_ptr()
    gemm.grouped_gemm_bf16(a, w, offs, epilogue=gemm.EPI_SCATTER_ROWS, row_info=perm.to(torch.int64), scatter_bases=bases,
                           scatter_row_bytes=n * 2, scatter_slots=total, tile_n=tile_n, w_prefetch=w_prefetch, tile_m=tile_m)
    torch.cuda.synchronize()
    default_status().check()
    start = 0
    for gi, sz in enumerate(sizes):
        if sz:
            x = a[start:start + sz].float()
            ref = x @ w[gi].float().t()
            _check(out[start:start + sz], ref, k)
            _check(dst[perm[start:start + sz]], ref, k)
            _check(h[start:start + sz], torch.nn.functional.silu(x @ w2[gi, :n].float().t()) * (x @ w2[gi, n:].float().t()), k)
        start += sz


@pytest.mark.parametrize("pair", [False, True, "wide", "swap"])
def test_grouped_gemm_scatter_rows(pair):
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(6)
    sizes = [40, 0, 200] + ([517] if pair else [])
    g, k, n = len(sizes), 256, 512
    total = sum(sizes)
    offs = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    a = torch.randn(total, k, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(g, n, k, device="cuda") * 0.05).to(torch.bfloat16)
    dst = torch.zeros(total, n, device="cuda", dtype=torch.bfloat16)
    perm = torch.randperm(total, device="cuda")
    import ctypes

    row_info = perm.to(torch.int64).clone()  # region 0, slot = destination row
    row_info[3] = -1  # dropped row (region index out of range)
    bases = (ctypes.c_ulonglong * 8)()
    bases[0] = dst.data_ptr()
    scale = torch.rand(total, device="cuda") + 0.5
    gemm.grouped_gemm_bf16(a, w, offs, epilogue=gemm.EPI_SCATTER_ROWS, row_info=row_info, scatter_bases=bases,
                           scatter_row_bytes=n * 2, scatter_slots=total, row_scale=scale, pair=pair)
    torch.cuda.synchronize()
    default_status().check()
    ref = torch.zeros(total, n, device="cuda")
    start = 0
    for gi, sz in enumerate(sizes):
        if sz:
            ref[start:start + sz] = (a[start:start + sz].float() @ w[gi].float().t()) * scale[start:start + sz, None]
        start += sz
    expect = torch.zeros_like(ref)
    expect[perm] = ref
    expect[perm[3]] = 0
    _check(dst, expect, k)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (512, 512, 512), (1000, 4096, 4096), (8192, 3584, 512), (4096, 1152, 256), (300, 4128, 192),
                                   (2048, 8192, 8192)])
def test_gemm_bf16_cta_pair(m, n, k, wide):
    """The cta_group::2 kernels (256-row tiles on two SMs; ``wide``: 256 x 512 tiles in two accumulator blocks): same
    product, ragged edges in M and N (a tile whose second block lies outside N), all tile widths, several bands of
    tile columns (the last one narrower)."""
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(m + n + k + 1)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = gemm.gemm_bf16_pair(a, b, wide=wide)
    torch.cuda.synchronize()
    default_status().check()
    ref = a.float() @ b.float().t()
    _check(out, ref, k)


@pytest.mark.parametrize("m,n,k", [(128, 256, 128), (256, 512, 1024), (1000, 3584, 2048), (300, 4128, 512)])
def test_gemm_fp8_blockscaled(m, n, k):
    """e4m3 x e4m3 with 1x128 activation scales and 128x128 weight scales against the fp32 product of the dequantised operands."""
    from dlslime_b200.ops import gemm, quant
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(m * 3 + n + k)
    a = (torch.randn(m, k, device="cuda") * torch.rand(m, 1, device="cuda") * 4).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    aq, sa = quant.fp8_quant_1x128(a)
    wq, sb = quant.fp8_quant_128x128(w)
    out = gemm.gemm_fp8_blockscaled(aq, sa, wq, sb)
    torch.cuda.synchronize()
    default_status().check()
    ref = gemm.ref_gemm_fp8_blockscaled(aq, sa, wq, sb)
    # same quantised operands on both sides: only fp32 summation order and the bf16 rounding of the output differ
    err = (out.float() - ref).abs().max().item()
    assert err <= 2e-2 * ref.abs().max().item() + 1e-3, err
    # and the product is a faithful fp8 approximation of the bf16 one
    full = a.float() @ w.float().t()
    rel = (out.float() - full).norm() / full.norm()
    assert rel < 0.08, rel.item()


def test_grouped_gemm_with_fp8_activations_is_bit_identical_to_dequant_then_gemm():
    """The gate/up GEMM fed with e4m3 rows and 1x128 scales (expanded in shared memory) against the two-pass path."""
    from dlslime_b200.ops import gemm, quant
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(11)
    sizes = [0, 5, 128, 131, 300, 1, 0, 64]
    g, k, inter = len(sizes), 1024, 256
    offs = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total = sum(sizes)
    x = (torch.randn(total + 37, k, device="cuda") * torch.rand(total + 37, 1, device="cuda") * 3).to(torch.bfloat16)
    xq, xs = quant.fp8_quant_1x128(x)
    xd = quant.fp8_dequant_1x128(xq, xs)
    w13 = (torch.randn(g, 2 * inter, k, device="cuda") * 0.05).to(torch.bfloat16)
    w = (torch.randn(g, inter, k, device="cuda") * 0.05).to(torch.bfloat16)
    for weights, epi in ((w13, gemm.EPI_SWIGLU), (w, gemm.EPI_STORE)):
        ref = torch.zeros((total + 37, inter), device="cuda", dtype=torch.bfloat16)
        out = torch.zeros_like(ref)
        gemm.grouped_gemm_bf16(xd, weights, offs, out=ref, epilogue=epi)
        gemm.grouped_gemm_fp8a(xq, xs, weights, offs, out=out, epilogue=epi)
        torch.cuda.synchronize()
        default_status().check()
        assert torch.equal(out[:total], ref[:total]), (out[:total].float() - ref[:total].float()).abs().max().item()
        assert bool((out[total:] == 0).all())


@pytest.mark.parametrize("tile_tokens", [64, 128, 192])
@pytest.mark.parametrize("sizes,n,k", [([3, 0, 130, 257, 64], 448, 384), ([1], 32, 64), ([16, 17, 128, 129, 192, 193, 385], 288, 1096), ([0, 0, 5], 1024, 512)])
def test_grouped_gemm_weights_on_the_m_side(sizes, n, k, tile_tokens):
    """Groups below, at and above one tile of tokens, empty ones, feature tiles that reach past N (into the next group and past the
    end), a K that is no multiple of 64; store, SwiGLU and scatter with row weights and dropped rows against the fp32 product."""
    import ctypes

    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(n + k + tile_tokens)
    g, total = len(sizes), sum(sizes)
    offs = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    a = torch.randn(total + 3, k, device="cuda", dtype=torch.bfloat16)  # rows behind the last group are nobody's
    w = (torch.randn(g, n, k, device="cuda") * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(g, 2 * n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((total + 3, n), 9.0, device="cuda", dtype=torch.bfloat16)
    gemm.grouped_gemm_bf16(a, w, offs, out=out, tile_tokens=tile_tokens)
    h = gemm.grouped_gemm_bf16(a, w2, offs, epilogue=gemm.EPI_SWIGLU, tile_tokens=tile_tokens)
    dst = torch.zeros(total, n, device="cuda", dtype=torch.bfloat16)
    perm = torch.randperm(total, device="cuda")
    info = torch.cat([perm, torch.zeros(3, dtype=torch.int64, device="cuda")])
    info[total // 2] = 5 << 48  # a region that does not exist: the row is dropped
    scale = torch.rand(total + 3, device="cuda")
    bases = (ctypes.c_ulonglong * 8)()
    bases[0] = dst.data_ptr()
    gemm.grouped_gemm_bf16(a, w, offs, epilogue=gemm.EPI_SCATTER_ROWS, row_info=info, row_scale=scale, scatter_bases=bases,
                           scatter_row_bytes=n * 2, scatter_slots=total, tile_tokens=tile_tokens)
    torch.cuda.synchronize()
    default_status().check()
    assert (out[total:] == 9.0).all() and (dst[perm[total // 2]] == 0).all()
    start = 0
    for gi, sz in enumerate(sizes):
        rows = slice(start, start + sz)
        if sz:
            x = a[rows].float()
            ref = x @ w[gi].float().t()
            keep = torch.arange(start, start + sz, device="cuda") != total // 2
            _check(out[rows], ref, k)
            if keep.any():
                _check(dst[perm[rows]][keep], (ref * scale[rows, None])[keep], k)
            _check(h[rows], torch.nn.functional.silu(x @ w2[gi, :n].float().t()) * (x @ w2[gi, n:].float().t()), k)
        start += sz


@pytest.mark.parametrize("m,n,k", [(1, 32, 128), (72, 4096, 7168), (72, 4096, 1024), (129, 2080, 384), (2400, 2048, 640), (3300, 2048, 256),
                                   (65, 8192, 1152), (300, 4128, 4096), (257, 288, 2304), (20000, 512, 512)])
def test_gemm_fp8_forms(m, n, k):
    """Single CTAs (one block of K), clusters of 2, 4 and 8 that share K unevenly, and CTA pairs with the last round cut into
    column parts (wide and narrow tiles in one launch, parts past the end of N, rows past M in one CTA of the pair)."""
    from dlslime_b200.ops import gemm, quant
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(m + 5 * n + k)
    a = (torch.randn(m, k, device="cuda") * (torch.rand(m, 1, device="cuda") + 0.1) * 4).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    aq, sa = quant.fp8_quant_1x128(a)
    wq, sb = quant.fp8_quant_128x128(w)
    out = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm_fp8_blockscaled(aq, sa, wq, sb, out=out[:m])
    torch.cuda.synchronize()
    default_status().check()
    blocks = sb.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    ref = (aq.double() * sa.double().repeat_interleave(128, 1)) @ (wq.double() * blocks).t()
    # bf16 rounding of the result (2^-9), and k fp32 additions of terms whose magnitudes sum to at most ~sqrt(k) results
    tol = ref.abs() * 2 ** -8 + ref.pow(2).mean().sqrt() * k ** 0.5 * 2 ** -20
    assert ((out[:m].double() - ref).abs() <= tol).all()
    assert (out[m] == 7.0).all(), "a row past the end was written"


@pytest.mark.parametrize("m,n,k", [(1, 32, 2048), (72, 4096, 7168), (129, 544, 4104), (300, 1056, 8192), (500, 2048, 2056), (128, 8192, 1984)])
def test_gemm_bf16_few_tiles_share_k(m, n, k):
    """Products with few output tiles: clusters of 2, 4 and 8 CTAs per tile, a K that they share unevenly, rows past M and tile
    columns past N; rows behind the last one stay."""
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm_bf16(a, b, out=out[:m])
    torch.cuda.synchronize()
    default_status().check()
    _check(out[:m], a.float() @ b.float().t(), k)
    assert (out[m] == 7.0).all()


@pytest.mark.parametrize("groups", [7, 256, 257, 300])
def test_grouped_gemm_weights_on_m_chained(groups):
    """Launches chained to the one in front: the second product fetches its first weights early (K of two blocks, less than the
    ring; up to 256 groups, whose prefix fits in shared memory) and reads rows that the launch in front of it writes. New
    rows every time, so that rows of an earlier pass would show; bit for bit what ordinary launches give."""
    from dlslime_b200.ops import gemm
    from dlslime_b200.ops._common import default_status

    gen = torch.Generator(device="cuda").manual_seed(groups)
    sizes = torch.randint(0, 70 if groups == 7 else 5, (groups,), generator=gen, device="cuda")
    offs = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), sizes.cumsum(0)]).to(torch.int32)
    total, mid, n = int(offs[-1]), 128, 160
    w1 = (torch.randn((groups, 2 * mid, 256), generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
    w2 = (torch.randn((groups, n, mid), generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
    h, out = torch.empty((total, mid), device="cuda", dtype=torch.bfloat16), torch.empty((total, n), device="cuda", dtype=torch.bfloat16)
    xs = [torch.randn((total, 256), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(6)]
    want = []
    for x in xs:
        gemm.grouped_gemm_bf16(x, w1, offs, out=h, epilogue=gemm.EPI_SWIGLU, tile_tokens=64)
        want.append(gemm.grouped_gemm_bf16(h, w2, offs, tile_tokens=64))
    torch.cuda.synchronize()
    got = []
    for x in xs:
        gemm.grouped_gemm_bf16(x, w1, offs, out=h, epilogue=gemm.EPI_SWIGLU, tile_tokens=64, chained=1)
        gemm.grouped_gemm_bf16(h, w2, offs, out=out, tile_tokens=64, chained=2)
        got.append(out.clone())
    torch.cuda.synchronize()
    default_status().check()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    x = xs[0].float()
    for gi in (0, groups // 2, groups - 1):
        r = slice(int(offs[gi]), int(offs[gi + 1]))
        if r.stop > r.start:
            g = (torch.nn.functional.silu(x[r] @ w1[gi, :mid].float().t()) * (x[r] @ w1[gi, mid:].float().t())).to(torch.bfloat16).float()
            _check(want[0][r], g @ w2[gi].float().t(), mid)


@pytest.mark.parametrize("m,k,shared", [(64, 1024, True), (65, 1024, True), (128, 1024, False), (128, 1472, True), (300, 1664, True), (300, 1472, False), (16, 832, False)])
def test_clusters_are_worth_more_k_blocks_for_taller_tiles(m, k, shared):
    """The launcher shares a tile's K where that saves 14 K blocks per CTA, 19 for tiles of 128 rows, whose sums are twice as many."""
    from dlslime_b200 import _lib

    assert (_lib.call("slime_gemm_bf16_clusters", m, 2048, k) > 1) is shared
    test_gemm_bf16_few_tiles_share_k(m, 2048, k)


@pytest.mark.parametrize("m,n,k", [(300, 8192, 4480), (300, 8192, 4608), (600, 3584, 4608), (701, 4320, 6912), (1000, 8192, 5632), (2300, 6144, 5760), (3000, 6144, 5632)])
def test_gemm_fp8_deep_products_of_few_rounds(m, n, k):
    """On both sides of the line between CTA pairs and single CTAs: one round below and from 36 K blocks, two and three rounds from 44, four
    rounds; ragged rows and columns."""
    test_gemm_fp8_forms(m, n, k)
