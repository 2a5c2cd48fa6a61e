"""KV pack / unpack / transfer kernels: bit-exact against torch index copies."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(prompt_lens, page=64, row=256, blocks=None):
    from dlslime_b200.ops import kv

    pages = sum((n + page - 1) // page for n in prompt_lens)
    blocks = blocks or pages + 7
    g = torch.Generator().manual_seed(3)
    dst_blocks = torch.randperm(blocks, generator=g)[:pages].tolist()
    tasks = kv.build_page_tasks(prompt_lens, page, dst_blocks)
    return tasks, dst_blocks, blocks


def test_pack_unpack_roundtrip_bit_exact():
    from dlslime_b200.ops import kv
    from dlslime_b200.ops._common import default_status

    lens, page, row = [100, 64, 1, 513, 129], 64, 256
    (tok_off, blk, ntok), dst_blocks, blocks = _setup(lens, page, row)
    total = sum(lens)
    src = torch.randn(2, total, row, device="cuda").to(torch.bfloat16)
    paged = torch.zeros(2, blocks, page, row, device="cuda", dtype=torch.bfloat16)
    kv.kv_pack(src, paged, tok_off, blk, ntok)
    torch.cuda.synchronize()
    default_status().check()
    expect = torch.zeros_like(paged)
    for t, b, n in zip(tok_off.tolist(), blk.tolist(), ntok.tolist()):
        expect[:, b, :n] = src[:, t:t + n]
    assert torch.equal(paged, expect)
    back = torch.zeros_like(src)
    kv.kv_unpack(paged, back, tok_off, blk, ntok)
    torch.cuda.synchronize()
    assert torch.equal(back, src)


def test_out_of_range_block_is_reported_not_written():
    from dlslime_b200.ops import kv
    from dlslime_b200.ops._common import default_status

    page, row = 64, 256
    src = torch.randn(2, 128, row, device="cuda").to(torch.bfloat16)
    paged = torch.zeros(2, 4, page, row, device="cuda", dtype=torch.bfloat16)
    tok_off = torch.tensor([0, 64], dtype=torch.int32, device="cuda")
    blk = torch.tensor([1, 9], dtype=torch.int32, device="cuda")  # block 9 does not exist
    kv.kv_pack(src, paged, tok_off, blk)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        default_status().check()
    assert torch.equal(paged[:, 1], src[:, :64]) and paged[:, [0, 2, 3]].abs().sum() == 0


def test_prefill_sender_pushes_every_layer_with_flags():
    """Emulated peer on one GPU: the 'decode' cache is a second region on the same device."""
    from dlslime_b200.models.pd_kv import KVShape, PagedKVCache, PrefillSender, wait_layers
    from dlslime_b200.ops._common import default_status
    from dlslime_b200.parallel.symm import SymmetricHeap

    shape = KVShape(layers=4, kv_heads_local=2, head_dim=128, page_tokens=64)
    lens = [130, 64, 700]
    pages = sum((n + 63) // 64 for n in lens)
    blocks = pages + 5
    heap = SymmetricHeap.emulated(2, PagedKVCache.bytes_needed(shape, blocks))
    cache = PagedKVCache(shape, blocks, heap, owner_rank=1)
    sender = PrefillSender(shape, cache, max_tokens=sum(lens), comm_blocks=16)
    g = torch.Generator().manual_seed(5)
    dst_blocks = torch.randperm(blocks, generator=g)[:pages].tolist()
    tok_off, blk, ntok = sender.plan(lens, dst_blocks)
    sender.kv_stage.copy_(torch.randn(sender.kv_stage.shape, device="cuda"))
    d = 256
    hidden = torch.randn(sum(lens), d, device="cuda").to(torch.bfloat16)
    weights = [(torch.randn(d, d, device="cuda") * 0.05).to(torch.bfloat16)]
    sender.run_prefill_with_transfer(hidden, weights, overlap=True)
    torch.cuda.synchronize()
    default_status().check()
    assert wait_layers(cache, sender.step, timeout_s=2.0)
    got = cache.tensor()
    for t, b, n in zip(tok_off.tolist(), blk.tolist(), ntok.tolist()):
        assert torch.equal(got[:, :, b, :n], sender.kv_stage[:, :, t:t + n])


@pytest.mark.parametrize("page,row,lens,threads", [(1, 8, [5, 1], 256), (7, 2056, [7, 20, 1], 256), (16, 128, [1000, 16, 3], 32), (64, 512, [63, 65, 640], 96), (64, 512, [63, 65, 640], 256),
                                                   (40, 1000, [41] * 40, 256)])
def test_page_sizes_that_are_no_multiple_of_a_slice(page, row, lens, threads):
    """Pages below, above and beside the 4 KB slices that a warp moves, from a page of 16 bytes on; short last pages, CTAs of
    one, three and eight warps, fewer CTAs than slices; nothing outside the pages' rows is written."""
    from dlslime_b200.ops import kv
    from dlslime_b200.ops._common import default_status

    (tok_off, blk, ntok), _, blocks = _setup(lens, page, row)
    total, rb = sum(lens), row * 2
    src = torch.randn(2, total, row, device="cuda").to(torch.bfloat16)
    paged = torch.full((2, blocks, page, row), 3.0, device="cuda", dtype=torch.bfloat16)
    expect = paged.clone()
    for t, b, n in zip(tok_off.tolist(), blk.tolist(), ntok.tolist()):
        expect[:, b, :n] = src[:, t:t + n]
    back = torch.full_like(src, 4.0)
    kv.tune(threads)
    try:
        for max_blocks in (0, 3):
            kv.kv_move(src[0].data_ptr(), src[1].data_ptr(), paged[0].data_ptr(), paged[1].data_ptr(), tok_off, blk, ntok,
                       page_tokens=page, row_bytes=rb, tok_rows=total, page_blocks=blocks, to_paged=True, max_blocks=max_blocks)
            kv.kv_move(back[0].data_ptr(), back[1].data_ptr(), paged[0].data_ptr(), paged[1].data_ptr(), tok_off, blk, ntok,
                       page_tokens=page, row_bytes=rb, tok_rows=total, page_blocks=blocks, to_paged=False, max_blocks=max_blocks)
            torch.cuda.synchronize()
            default_status().check()
            assert torch.equal(paged, expect) and torch.equal(back, src)
            paged.fill_(3.0)
            back.fill_(4.0)
    finally:
        kv.tune(256)


@pytest.mark.parametrize("form,threads", [("registers", 0), ("registers", 96), ("bulk", 0), ("auto", 64)])
@pytest.mark.parametrize("page,row,lens", [(1, 8, [5, 1]), (64, 256, [63, 65, 640]), (64, 4104, [64, 129, 1])])
def test_every_form_moves_the_same_bytes(page, row, lens, form, threads):
    """The form a call names, for pages below, at and above one bulk chunk (16 B, 32 KB, 513 KB), with short last pages."""
    from dlslime_b200.ops import kv
    from dlslime_b200.ops._common import default_status

    (tok_off, blk, ntok), _, blocks = _setup(lens, page, row)
    total, rb = sum(lens), row * 2
    src = torch.randn(2, total, row, device="cuda").to(torch.bfloat16)
    paged = torch.full((2, blocks, page, row), 3.0, device="cuda", dtype=torch.bfloat16)
    expect, back = paged.clone(), torch.full_like(src, 4.0)
    for t, b, n in zip(tok_off.tolist(), blk.tolist(), ntok.tolist()):
        expect[:, b, :n] = src[:, t:t + n]
    for to_paged, tok in ((True, src), (False, back)):
        kv.kv_move(tok[0].data_ptr(), tok[1].data_ptr(), paged[0].data_ptr(), paged[1].data_ptr(), tok_off, blk, ntok, page_tokens=page,
                   row_bytes=rb, tok_rows=total, page_blocks=blocks, to_paged=to_paged, max_blocks=5, form=form, threads=threads)
    torch.cuda.synchronize()
    default_status().check()
    assert torch.equal(paged, expect) and torch.equal(back, src)
