"""Scratch memory of the native FastConformer calls on the host side: which buffer a call in flight holds (no GPU)."""
import ctypes

import torch

from oasr_b200 import _lib, functional
from oasr_b200.fastconformer import FastConformerLayers
from oracle import fastconformer as OFC

CFG = OFC.FastConformerConfig(hidden=256, heads=2, ffn=512, layers=2, kernel=9, sliding_window=25, lookahead=3, bias=True)


def _address(arg):
    return arg.value if isinstance(arg, ctypes.c_void_p) else arg


def test_a_streaming_step_shares_its_scratch_with_no_other_call_in_flight(monkeypatch):
    """A step on another CUDA stream or thread is enqueued while the first one runs: neither its scratch nor that of a packed
    batch may overlap.  The second and third call are made from inside the first, whose scratch is then certainly held."""
    model = FastConformerLayers(CFG.hidden, CFG.heads, CFG.ffn, CFG.layers, CFG.kernel, CFG.sliding_window, CFG.lookahead,
                                OFC.init_params(CFG, 5), device="cpu")
    cache = model.new_streaming_cache(4)
    held, names = [], []

    def step(streams):
        table, cached, _, pos_start, slots = cache.prepare(streams)
        model._chunk_native(torch.zeros(len(streams) * 16, CFG.hidden), len(streams), 16, cache, table, cached, pos_start, slots)

    def packed():
        cu = torch.tensor([0, 8], dtype=torch.int32)
        g = {"T": 8, "cu": cu, "offsets": torch.tensor([0, 128]), "bias_numel": 128}
        model._layers_native(torch.zeros(8, CFG.hidden), g)

    def record(name, *args):
        nested = not names
        names.append(name)
        held.append((_address(args[-3]), args[-2]))           # workspace, its bytes, stream
        if nested:
            step([3])
            packed()

    monkeypatch.setattr(functional, "_stream", lambda t: None)
    monkeypatch.setattr(_lib, "call", record)
    step([0, 1, 2])
    assert names == ["oasr_b200_fastconformer_chunk_paged"] * 2 + ["oasr_b200_fastconformer_layers_packed"]
    spans = sorted((at, at + size) for at, size in held)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:])), spans


def test_native_step_takes_only_caches_of_its_own_type_and_geometry():
    """The native step passes the pools by address, so it may not be given one whose elements or extents differ; pools of other
    layer strides are fine."""
    from oasr_b200.streaming import StreamingCache

    model = FastConformerLayers(CFG.hidden, CFG.heads, CFG.ffn, CFG.layers, CFG.kernel, CFG.sliding_window, CFG.lookahead,
                                OFC.init_params(CFG, 5), device="cpu")
    make = lambda layers=2, heads=2, dim=128, width=256, kernel=9, **kw: StreamingCache(
        layers, heads, dim, width, kernel, 4, 32, device="cpu", **{"dtype": torch.bfloat16, **kw})
    assert model._native_cache(model.new_streaming_cache(4)) and model._native_cache(make(layers=3))
    assert not model._native_cache(make(dtype=torch.float16))
    assert not model._native_cache(make(kv_scales=torch.ones(2, 2, 2)))          # one byte per element
    assert not model._native_cache(make(heads=1)) and not model._native_cache(make(dim=64)) and not model._native_cache(make(layers=1))
    assert not model._native_cache(make(width=128)) and not model._native_cache(make(kernel=15))
    spread = make()
    spread.k_pool, spread.v_pool = (torch.zeros(4, *p.shape[1:], dtype=p.dtype)[::2] for p in (spread.k_pool, spread.v_pool))
    assert model._native_cache(spread)
    assert spread.pool_pointers()[0][1] == spread.k_pool[1].data_ptr() and spread.pool_pointers()[1][1] == spread.v_pool[1].data_ptr()
    spread.v_pool = spread.v_pool.transpose(2, 3).contiguous().transpose(2, 3)
    assert not model._native_cache(spread)
