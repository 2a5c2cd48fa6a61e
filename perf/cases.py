"""The work that a program using this package has it do on one GPU, as cases that can be timed and compared.

Six families, each through the public entry points:

* ``moe``       one step of :class:`ExpertParallelMoE` (route, dispatch, expert FFN, combine), launched eagerly or
                replayed from the layer's CUDA graph;
* ``prefill``   the prefill side of a disaggregated server: the per-layer GEMM chain with every layer's KV pages sent to
                the decode cache while the next layer computes;
* ``kv``        the paged KV movement by itself: a whole batch planned and pushed layer by layer, or one layer packed or
                unpacked on the decode side;
* ``linear``    a linear layer on the tensor cores, bf16 or block-scaled fp8 (activations quantised in the call);
* ``quant``     1x128 quantisation of activations and the way back;
* ``endpoint``  batched one-sided reads and writes of the NVLink endpoint, both regions on this GPU.

Sizes are those of the package's benchmark and tests (the 256-expert MoE layer with hidden 7168 and intermediate 2048,
the 32-layer KV shape with 64-token pages, the tensor-parallel [8192, 8192] x [8192, 28672 / 8] product, batches of 4096
pieces of 64 KiB), and ragged ones in between.
"""

import math

import torch

from dlslime_b200.models.moe import ExpertParallelMoE, MoEConfig, init_expert_weights
from dlslime_b200.models.pd_kv import KVShape, PagedKVCache, PrefillSender
from dlslime_b200.ops import gemm, kv, quant
from dlslime_b200.ops.nvlink import NVLinkEndpoint
from dlslime_b200.parallel.symm import SymmetricHeap

MODEL_DIM = 4096  # width of the GEMM that stands for a layer's compute in the prefill chain


def listed():
    return [
        # The headline step: prefill of 4096 tokens, all 256 experts on this GPU, about 128 rows per expert.
        {"name": "moe_prefill_256e", "kind": "moe", "experts": 256, "topk": 8, "hidden": 7168, "inter": 2048, "tokens": 4096,
         "graph": False, "renormalize": False},
        # What one of eight ranks computes in that step: 32 experts with about 1024 rows each.
        {"name": "moe_prefill_32e", "kind": "moe", "experts": 32, "topk": 8, "hidden": 7168, "inter": 2048, "tokens": 4096,
         "graph": False, "renormalize": False},
        # One of eight ranks in a decode step of 128 tokens, replayed from the layer's graph: about 32 rows per expert.
        {"name": "moe_decode_32e_graph", "kind": "moe", "experts": 32, "topk": 8, "hidden": 7168, "inter": 2048, "tokens": 128,
         "graph": True, "renormalize": False},
        # A chunked prefill or mixed batch on one of four ranks: a ragged token count, renormalised gates.
        {"name": "moe_mixed_64e", "kind": "moe", "experts": 64, "topk": 8, "hidden": 7168, "inter": 2048, "tokens": 777,
         "graph": False, "renormalize": True},
        # The smallest step: three sequences decoding, launched eagerly.
        {"name": "moe_decode_3tok", "kind": "moe", "experts": 32, "topk": 8, "hidden": 7168, "inter": 2048, "tokens": 3,
         "graph": False, "renormalize": False},
        # The prefill rank at work: 16 prompts of 512 to 8192 tokens, 32 layers, transfer under the compute.
        {"name": "prefill_16_prompts", "kind": "prefill", "batch": 7, "prompts": 16, "shortest": 512, "longest": 8192, "layers": 32,
         "heads": 2, "page": 64, "blocks": 32},
        # Only the hand-off, for a server whose compute is elsewhere: five prompts, planned and pushed for all layers.
        {"name": "kv_push_5_prompts", "kind": "kv", "op": "push", "batch": 8, "prompts": 5, "shortest": 512, "longest": 8192, "layers": 32,
         "heads": 2, "page": 64, "blocks": 32},
        # The tensor-parallel projection of the fp8 all-gather benchmark on one rank, with its activations' quantisation.
        {"name": "linear_fp8_8192", "kind": "linear", "dtype": "fp8", "m": 8192, "n": 3584, "k": 8192},
        # A decode-size projection in fp8: few rows, so there are far fewer tiles than SMs.
        {"name": "linear_fp8_72", "kind": "linear", "dtype": "fp8", "m": 72, "n": 4096, "k": 7168},
        # Activations to the wire format and back, a ragged number of rows.
        {"name": "quant_roundtrip", "kind": "quant", "rows": 12289, "cols": 7168},
        # 4096 pieces of 64 KiB from permuted places of a 4 GiB region.
        {"name": "endpoint_read_scatter", "kind": "endpoint", "op": "read", "pieces": 4096, "length": 65536, "align": 65536,
         "region": 4 << 30, "wait": False},
        # A small control-plane write whose sender waits for it: a few unaligned pieces.
        {"name": "endpoint_write_small", "kind": "endpoint", "op": "write", "pieces": 24, "length": 3001, "align": 1,
         "region": 1 << 20, "wait": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["moe", "moe", "moe", "prefill", "kv", "linear", "linear", "quant", "endpoint"])
    if kind == "moe":
        hidden, inter = rng.choice([(7168, 2048), (7168, 2048), (4096, 1024), (1024, 256)])
        tokens = _log_int(rng, 1, 4096)
        return {"kind": "moe", "experts": rng.choice([32, 64, 128, 256]), "topk": rng.choice([4, 8, 8]), "hidden": hidden,
                "inter": inter, "tokens": tokens, "graph": tokens <= 256 and rng.random() < 0.5, "renormalize": rng.random() < 0.5}
    if kind in ("prefill", "kv"):
        case = {"kind": kind, "batch": rng.randrange(1 << 20), "prompts": rng.randint(1, 16), "shortest": _log_int(rng, 16, 512), "longest": _log_int(rng, 600, 8192),
                "layers": rng.choice([8, 16, 32]), "heads": rng.choice([1, 2, 4]), "page": rng.choice([16, 64, 64]),
                "blocks": rng.choice([32, 148])}
        if kind == "kv":
            case["op"] = rng.choice(["push", "pack", "unpack"])
        return case
    if kind == "linear":
        return {"kind": "linear", "dtype": rng.choice(["bf16", "fp8"]), "m": _log_int(rng, 1, 8192), "n": 32 * _log_int(rng, 16, 256),
                "k": 128 * _log_int(rng, 8, 64)}
    if kind == "quant":
        return {"kind": "quant", "rows": _log_int(rng, 1, 32768), "cols": 128 * _log_int(rng, 8, 64)}
    pieces = _log_int(rng, 1, 4096)
    align = rng.choice([1, 16, 4096])
    length = _log_int(rng, 8, 65536)
    if align > 1:
        length = -(-length // 16) * 16
    return {"kind": "endpoint", "op": rng.choice(["read", "write"]), "pieces": pieces, "length": length, "align": align,
            "region": max(1 << 20, 2 * pieces * max(align, length + align)), "wait": rng.random() < 0.5}


def _prompt_lens(case):
    g = torch.Generator().manual_seed(case["batch"])  # which batch of prompts: part of the case, the seed fills it
    return torch.randint(case["shortest"], case["longest"] + 1, (case["prompts"],), generator=g).tolist()




def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0):
        out = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        return out.normal_(0.0, std, generator=gen)

    kind = case["kind"]
    st = {"case": case}
    if kind == "moe":
        cfg = MoEConfig(num_experts=case["experts"], topk=case["topk"], hidden=case["hidden"], intermediate=case["inter"],
                        renormalize=case["renormalize"])
        weights = init_expert_weights(cfg, range(cfg.num_experts), torch.device("cuda"), seed)
        st["layer"] = ExpertParallelMoE(cfg, max_tokens=case["tokens"], weights=weights)
        st["x"] = normal(case["tokens"], cfg.hidden)
        st["logits"] = torch.randn((case["tokens"], cfg.num_experts), generator=gen, device="cuda")
        if case["graph"]:
            st["x_in"], st["logits_in"], st["out"] = st["x"].clone(), st["logits"].clone(), torch.empty_like(st["x"])
            st["step"] = st["layer"].capture(st["x_in"], st["logits_in"], st["out"])
    elif kind in ("prefill", "kv"):
        lens = _prompt_lens(case)
        one_layer = case.get("op") in ("pack", "unpack")
        shape = KVShape(layers=1 if one_layer else case["layers"], kv_heads_local=case["heads"], page_tokens=case["page"])
        pages = sum(-(-n // shape.page_tokens) for n in lens)
        tokens, blocks = sum(lens), pages + 64
        # the decode side's block table: a random choice of free blocks
        table = torch.randperm(blocks, generator=torch.Generator().manual_seed(seed + 1))[:pages].tolist()
        if one_layer:
            st["tasks"] = kv.build_page_tasks(lens, shape.page_tokens, table)
            st["tokens_kv"] = normal(2, tokens, shape.row)
            st["paged_kv"] = normal(2, blocks, shape.page_tokens, shape.row)
        else:
            heap = SymmetricHeap(PagedKVCache.bytes_needed(shape, blocks))
            st["cache"] = PagedKVCache(shape, blocks, heap, owner_rank=0)
            st["sender"] = PrefillSender(shape, st["cache"], max_tokens=tokens, comm_blocks=case["blocks"])
            st["sender"].kv_stage.normal_(generator=gen)
            st["lens"], st["table"] = lens, table
            # what the decode side reads; the views do not own the heap's memory, so they carry it
            st["landed"] = (st["cache"].tensor(), st["cache"].layer_done())
            for view in st["landed"]:
                view.heap = heap
        if kind == "prefill":
            st["hidden"] = normal(tokens, MODEL_DIM)
            st["weights"] = [normal(MODEL_DIM, MODEL_DIM, std=MODEL_DIM ** -0.5) for _ in range(2)]
    elif kind == "linear":
        st["x"] = normal(case["m"], case["k"])
        w = normal(case["n"], case["k"], std=0.02)
        st["w"] = quant.fp8_quant_128x128(w) if case["dtype"] == "fp8" else w
    elif kind == "quant":
        st["x"] = normal(case["rows"], case["cols"])
    elif kind == "endpoint":
        n, length, align = case["pieces"], case["length"], case["align"]
        pitch = -(-length // align) * align
        far = torch.randint(0, 256, (case["region"],), dtype=torch.uint8, device="cuda", generator=gen)
        near = torch.randint(0, 256, (max(pitch * n, 16),), dtype=torch.uint8, device="cuda", generator=gen)
        a, b = NVLinkEndpoint(), NVLinkEndpoint()
        a.register_memory_region(near.data_ptr(), 0, near.numel(), "buf")
        b.register_memory_region(far.data_ptr(), 0, far.numel(), "buf")
        a.connect(b.endpoint_info())
        lh, rh = a.get_mr_handle("buf"), a.get_remote_mr_handle("buf")
        # every piece at its own place: slots of the far region, in random order, shifted inside the slot where it may be
        g = torch.Generator().manual_seed(seed)
        slots = case["region"] // (pitch + (align if align == 1 else 0))
        places = torch.randperm(slots, generator=g)[:n].tolist()
        step = case["region"] // slots // align * align
        st.update(near=near, far=far, ep=a, peer=b, assign=[(lh, rh, p * step, i * pitch, length) for i, p in enumerate(places)])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "moe":
        if not case["graph"]:
            return st["layer"](st["x"], st["logits"])
        st["x_in"].copy_(st["x"])
        st["logits_in"].copy_(st["logits"])
        st["step"].replay()
        return st["out"]
    if kind == "prefill":
        st["sender"].plan(st["lens"], st["table"])
        # the chain uses its input as scratch: every batch comes in a buffer of its own
        out = st["sender"].run_prefill_with_transfer(st["hidden"].clone(), st["weights"])
        return out, *st["landed"]
    if kind == "kv":
        if case["op"] == "push":
            st["sender"].plan(st["lens"], st["table"])
            for layer in range(case["layers"]):
                st["sender"].send_layer(layer)
            return st["landed"]
        if case["op"] == "pack":
            kv.kv_pack(st["tokens_kv"], st["paged_kv"], *st["tasks"])
            return st["paged_kv"]
        kv.kv_unpack(st["paged_kv"], st["tokens_kv"], *st["tasks"])
        return st["tokens_kv"]
    if kind == "linear":
        if case["dtype"] == "bf16":
            return gemm.gemm_bf16(st["x"], st["w"])
        q, s = quant.fp8_quant_1x128(st["x"])
        return gemm.gemm_fp8_blockscaled(q, s, *st["w"])
    if kind == "quant":
        q, s = quant.fp8_quant_1x128(st["x"])
        return q.view(torch.uint8), s, quant.fp8_dequant_1x128(q, s)
    future = (st["ep"].read if case["op"] == "read" else st["ep"].write)(st["assign"])
    if case["wait"] and future.wait() != 0:
        raise RuntimeError("the transfer did not complete")
    return st["near"] if case["op"] == "read" else st["far"]


def work(case):
    kind = case["kind"]
    if kind == "moe":
        t, e, k, h, i = case["tokens"], case["experts"], case["topk"], case["hidden"], case["inter"]
        hit = e * (1.0 - (1.0 - k / e) ** t)  # experts that at least one of the tokens is routed to, on average
        return {"bytes": hit * 3 * h * i * 2 + t * (4 * h + 4 * e), "flops": 2.0 * t * k * 3 * h * i}
    if kind in ("prefill", "kv"):
        t, row = sum(_prompt_lens(case)), case["heads"] * 128 * 2
        layers = 1 if case.get("op") in ("pack", "unpack") else case["layers"]
        moved = 2.0 * layers * 2 * t * row  # K and V, read once and written once
        if kind == "kv":
            return {"bytes": moved, "flops": 0}
        return {"bytes": moved + layers * (2 * t * MODEL_DIM * 2 + MODEL_DIM * MODEL_DIM * 2), "flops": layers * 2.0 * t * MODEL_DIM * MODEL_DIM}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + (1 if case["dtype"] == "fp8" else 2) * n * k + 2 * m * n, "flops": 2.0 * m * n * k}
    if kind == "quant":
        return {"bytes": case["rows"] * case["cols"] * (2 + 1 + 2 + 8 / 128), "flops": 0}
    return {"bytes": 2.0 * case["pieces"] * case["length"], "flops": 0}


def tolerance(case):
    # Against fp64 arithmetic on the same fp8 operands, the bf16 roundings of the outputs (and, for the layer and the
    # chain, of the intermediate activations) alone give 1.7e-3 (linear), 3.6e-3 (MoE step) and 9.4e-3 (32 layers).
    kind = case["kind"]
    if kind == "moe":
        return {"rel": 1e-2}
    if kind == "prefill":
        return {"rel": 2e-2}
    if kind == "linear":
        return {"rel": 7e-3}
    return "exact"


def _e4m3_groups(x):
    """x [rows, cols] bf16 in the wire format, e4m3 with one fp32 scale per 128 elements, as the fp64 values it stands for.
    The format is part of the path's definition, so the 64-bit results start from its values."""
    g = x.float().reshape(x.shape[0], -1, 128)
    amax = g.abs().amax(dim=-1, keepdim=True).clamp_min(1e-4)
    top = torch.full_like(amax, 448.0)
    q = (g * (top / amax)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return (q.double() * (amax / top).double()).reshape(x.shape)


def exact(case, seed):
    """What ``run`` returns for these inputs in 64-bit arithmetic, without the bf16 roundings on the way; ``None`` for
    what is only moved."""
    kind = case["kind"]
    if kind not in ("moe", "linear", "prefill"):
        return None
    st = prepare(case, seed)
    if kind == "linear":
        if case["dtype"] == "bf16":
            return st["x"].double() @ st["w"].double().t()
        q, s = st["w"]
        blocks = s.double().repeat_interleave(128, 0)[: case["n"]].repeat_interleave(128, 1)[:, : case["k"]]
        return _e4m3_groups(st["x"]) @ (q.double() * blocks).t()
    if kind == "prefill":
        a = st["hidden"].double()
        weights = [w.double() for w in st["weights"]]
        for layer in range(case["layers"]):
            a = a @ weights[layer % len(weights)].t()
        return a, None, None
    layer, inter = st["layer"], case["inter"]
    gates, picked = torch.topk(torch.softmax(st["logits"].double(), dim=-1), case["topk"], dim=-1)
    if case["renormalize"]:
        gates = gates / gates.sum(-1, keepdim=True)
    x = _e4m3_groups(st["x"])
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        tok, k = (picked == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        gate_up = x[tok] @ layer.w_gate_up[e].double().t()
        h = torch.nn.functional.silu(gate_up[:, :inter]) * gate_up[:, inter:]
        out.index_add_(0, tok, gates[tok, k].unsqueeze(1) * (h @ layer.w_down[e].double().t()))
    return out
