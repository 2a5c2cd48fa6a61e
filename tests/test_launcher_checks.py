"""Arguments that a kernel could not handle are refused by the launchers before anything is launched, so these calls need no GPU."""
import ctypes

import pytest

from dlslime_b200 import _lib

A, B, OUT, OFFS = 1 << 20, 2 << 20, 3 << 20, 4 << 20  # addresses that nothing dereferences
M, N, K = 300, 2048, 512

PLAIN = ["slime_gemm_bf16", "slime_gemm_bf16_pair", "slime_gemm_bf16_wide"]
GROUPED = ["slime_grouped_gemm_bf16", "slime_grouped_gemm_bf16_pair", "slime_grouped_gemm_bf16_wide", "slime_grouped_gemm_bf16_swapped"]


def _refused(name, *args):
    if not _lib.available():
        pytest.skip("kernel library not built")
    with pytest.raises(_lib.SlimeCudaError, match="aligned"):
        _lib.call(name, *args)


@pytest.mark.parametrize("shift", [2, 4])
@pytest.mark.parametrize("name", PLAIN)
def test_plain_products_refuse_an_output_between_two_vectors(name, shift):
    _refused(name, A, B, OUT + shift, M, N, K, K, K, N, None, None)


@pytest.mark.parametrize("shift", [2, 4])
def test_fp8_product_refuses_an_output_between_two_vectors(shift):
    import dlslime_b200.ops.gemm  # noqa: F401 (declares the launcher)

    _refused("slime_gemm_fp8_blockscaled", A, A, B, B, OUT + shift, M, N, K, K, K, N, None, None)


@pytest.mark.parametrize("ldc,shift", [(N, 4), (N + 1, 0), (N, 2)])
@pytest.mark.parametrize("name", GROUPED)
@pytest.mark.parametrize("epilogue", [0, 1])
def test_grouped_products_refuse_rows_between_two_vectors(name, epilogue, ldc, shift):
    bases = (ctypes.c_ulonglong * 8)()
    _refused(name, A, B, OUT + shift, OFFS, 4, M, N, K, K, K, ldc, epilogue, None, bases, 0, 0, None, None, None)


@pytest.mark.parametrize("form,threads,say", [(3, 0, "unknown form"), (-1, 0, "unknown form"), (1, 33, "threads per CTA"), (1, 288, "threads per CTA")])
def test_kv_transfer_refuses_forms_and_ctas_it_does_not_have(form, threads, say):
    import dlslime_b200.ops.kv  # noqa: F401 (declares the launcher)

    if not _lib.available():
        pytest.skip("kernel library not built")
    with pytest.raises(_lib.SlimeCudaError, match=say):
        _lib.call("slime_kv_transfer_form", A, A, B, B, OFFS, OFFS, None, 1, 64, 512, 64, 4, 1, None, 0, None, 0, form, threads, None, None)


@pytest.mark.parametrize("rank,under_compute", [(0, "auto"), (1, "registers")])
@pytest.mark.parametrize("threads", [256, 64])
def test_prefill_transfer_under_compute_names_its_form(monkeypatch, threads, rank, under_compute):
    """Under the GEMM chain a sender to another GPU asks for CTAs without shared memory; otherwise the form is left to the launcher's
    rule. Always with the sender's own CTAs, whatever other senders of the process have."""
    import contextlib

    import torch

    from dlslime_b200.models import pd_kv

    moves = []
    stream = type("S", (), {"wait_stream": lambda self, other: None, "cuda_stream": 0})()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: stream)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "Stream", lambda *a, **k: stream)
    real_empty, real_zeros = torch.empty, torch.zeros
    monkeypatch.setattr(torch, "empty", lambda *a, **k: real_empty(*a, **{**k, "device": "cpu"}))
    monkeypatch.setattr(torch, "zeros", lambda *a, **k: real_zeros(*a, **{**k, "device": "cpu"}))
    monkeypatch.setattr(pd_kv.gemm, "gemm_bf16", lambda a, w, out=None: out)
    monkeypatch.setattr(pd_kv.kv, "kv_move", lambda *a, **k: moves.append((k["form"], k["threads"])))
    monkeypatch.setattr(pd_kv.kv, "tune", lambda t: moves.append(("tuned the process", t)))
    cache = type("C", (), {"plane_addr": lambda self, *a: 0, "flag_addr": lambda self, layer: 0, "num_blocks": 4, "owner": 0,
                           "heap": type("H", (), {"rank": rank})})()
    sender = pd_kv.PrefillSender(pd_kv.KVShape(layers=2), cache, max_tokens=64, comm_threads=threads)
    sender.tasks = (None, None, None)
    sender.send_layer(0)
    hidden = real_empty(64, 8)
    sender.run_prefill_with_transfer(hidden, [hidden], overlap=True)
    sender.run_prefill_with_transfer(hidden, [hidden], overlap=False)
    assert moves == [("auto", threads)] + 2 * [(under_compute, threads)] + 2 * [("auto", threads)]
