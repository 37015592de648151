"""Workspace buffers on the CPU: which are kept, which are let go, and what happens when the device is short of memory; and which steps
ask for the largest of them, and which go through recurrences in chunks."""
import threading
import types

import torch

from tiny_inference_engine_b200.engine.workspace import Workspace
from tiny_inference_engine_b200.ops import gemm_select
from tiny_inference_engine_b200.parts import latent_attention
from tiny_inference_engine_b200.parts.model import Model


def test_spare_buffers_are_outgrown_without_a_trace_and_refused_when_memory_is_short(monkeypatch):
    monkeypatch.setattr(Workspace, "_free_bytes", lambda self: 8000)
    ws = Workspace(8, "cpu")
    a = ws.spare("x", 100, torch.bfloat16, 128)
    assert a.numel() == 128 and ws.spare("x", 128, torch.bfloat16, 500) is a
    b = ws.spare("x", 129, torch.bfloat16, 1000)
    assert b.numel() == 1000 and ws.bytes() == 2000                # the outgrown one is gone
    assert ws.spare("x", 1001, torch.bfloat16, 2001) is None       # 4,002 bytes: more than half of what was left
    assert ws.spare("x", 1000, torch.bfloat16) is b                # what is there stays
    full = torch.empty

    def short(*a, **k):
        raise torch.cuda.OutOfMemoryError("no more")
    monkeypatch.setattr(torch, "empty", short)
    assert ws.spare("x", 1500, torch.bfloat16) is None and ws.bytes() == 0
    monkeypatch.setattr(torch, "empty", full)
    assert ws.spare("x", 1500, torch.bfloat16) is None             # not tried again at every step
    assert ws.spare("x", 1000, torch.bfloat16).numel() == 1000
    kept = ws.flat("y", 10, torch.float32)
    ws.flat("y", 11, torch.float32)
    assert ws.bytes() == 2000 + 40 + 80 and kept.numel() == 10     # a captured graph may still use it


def test_expanded_keys_stay_within_their_bytes():
    for heads, key_dim in ((1, 128), (16, 576), (32, 576), (33, 576), (64, 320), (128, 576), (500, 512)):
        keys = latent_attention.expanded_capacity(heads, key_dim)
        assert 0 < keys <= latent_attention.EXPAND_MAX_KEYS
        assert keys * 2 * (heads * 256 + key_dim) <= latent_attention.EXPAND_MAX_BYTES
    assert latent_attention.expanded_capacity(32, 576) == 16384 and latent_attention.expanded_capacity(128, 576) == 4528


def test_latents_are_multiplied_out_where_many_queries_share_a_key():
    pays = latent_attention.expanding_pays
    assert pays([64], [64], 0) == 64 and pays([2048], [2048], 0) == 2048 and pays([16384], [64], 0) == 16384
    assert pays([500] * 32, [2] * 32, 0) == 0 and pays([1000] * 16, [8] * 16, 0) == 0 and pays([500] * 16, [16] * 16, 0) == 0
    assert pays([300] * 4, [24] * 4, 0) == 4 * 320
    for context, n, window in ((70, 64, 0), (300, 64, 100), (90, 64, 40), (130, 64, 100), (5000, 65, 1024), (64, 64, 1)):
        pairs = sum(min(i + 1, window or 1 << 30) for i in range(context - n, context))
        rows = latent_attention.ops.latent_expanded_rows([context], [n], window)
        keys = context - max(0, context - n - window + 1 if window else 0)
        assert pays([context], [n], window) == (rows if pairs >= latent_attention.EXPAND_PAIRS_PER_KEY * keys else 0), (context, n, window)


def test_recurrences_go_in_chunks_where_that_was_measured_to_be_faster():
    from tiny_inference_engine_b200.ops import chunks_pay

    def pays(mode, lens, heads, dim, vdim):
        return chunks_pay(max(lens), len(lens), len(lens) * heads * -(-vdim // 16), dim, mode != "delta", mode == "head")
    assert not pays("delta", [64], 16, 128, 128) and not pays("delta", [96], 8, 128, 256) and not pays("delta", [128] + [1] * 30, 16, 128, 128)
    assert pays("delta", [128], 16, 64, 64) and pays("delta", [2048], 16, 128, 128) and pays("delta", [160] * 8, 16, 128, 128)
    assert not pays("channel", [96], 16, 128, 128) and not pays("channel", [128], 16, 64, 64) and not pays("channel", [128] * 2, 16, 64, 64)
    assert pays("channel", [128], 16, 128, 128) and pays("channel", [256], 16, 64, 64) and pays("channel", [160] * 8, 16, 64, 64)
    for lens, heads, dim, vdim in (([256], 16, 128, 128), ([2048], 16, 128, 128), ([4096], 32, 128, 64), ([2048], 32, 64, 64), ([96], 32, 128, 128),
                                   ([200] * 4, 16, 64, 64)):
        assert not pays("head", lens, heads, dim, vdim), (lens, heads, dim, vdim)
    for lens, heads, dim, vdim in (([2048], 32, 128, 128), ([1021, 510], 16, 128, 128), ([128] * 3, 16, 128, 128), ([1024] + [1] * 8, 16, 64, 64),
                                   ([1021] * 2, 64, 64, 64), ([256], 64, 128, 128), ([128] * 2, 64, 64, 64), ([128], 32, 128, 128)):
        assert pays("head", lens, heads, dim, vdim), (lens, heads, dim, vdim)


def test_sums_of_split_products_are_no_other_engines_memory():
    """Two engines stepping in two threads: a split product whose caller brings no memory uses the step's workspace; outside a step,
    memory that nothing else holds."""
    class Step(Model):
        def __init__(self):
            pass

        def _forward(self, ctx, cache, states):
            first = gemm_select._scratch_for(100, "cpu")
            meet.wait(10)                       # both steps are between their product and its reduction
            return first, gemm_select._scratch_for(200, "cpu")

    meet, got = threading.Barrier(2), {}
    spaces = [Workspace(4, "cpu") for _ in range(2)]

    def engine(i):
        got[i] = Step().forward(types.SimpleNamespace(ws=spaces[i]), None, None)
    threads = [threading.Thread(target=engine, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got[0][0] is got[0][1] and got[1][0] is got[1][1] and got[0][0].data_ptr() != got[1][0].data_ptr()
    assert spaces[0].flat("gemm.partial", 1, torch.float32) is got[0][0]
    outside = [gemm_select._scratch_for(100, "cpu") for _ in range(2)]
    assert outside[0].data_ptr() != outside[1].data_ptr()
