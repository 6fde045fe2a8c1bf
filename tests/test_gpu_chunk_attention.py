"""Attention and page append inside the native streaming step, through the C entry points, at page sizes, chunk lengths and
append positions that the Python cache never produces: against fp32 on the step's own projected queries, keys and values."""
import ctypes

import numpy as np
import pytest
import torch

import oasr_b200 as ob
from oasr_b200 import _lib
from oasr_b200.encoder import ConformerCTC, ConformerConfig
from oracle import conformer as OC

pytestmark = pytest.mark.gpu
CFG = OC.TINY_STREAM
ENTRIES = ["oasr_b200_conformer_chunk_paged", "oasr_b200_conformer_chunk_paged_split"]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _step(entry, model, rows, B, T, k_pools, v_pools, table, cached, total, pos_start, scales, cnn_state):
    """One native step.  Returns the last layer's projections (B, T, 4 d) and attention output (B, T, d), which the step leaves
    in its scratch: fp32 residual, h, y, FFN, projections, attention, ..., each padded to 256 bytes."""
    d, M = CFG.d_model, B * T
    need = _lib.load().oasr_b200_conformer_chunk_workspace_bytes(ctypes.byref(model._native_model), B, T)
    scratch = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    base = -scratch.data_ptr() % 256
    slots = torch.arange(B, device="cuda")
    pools = lambda ps: (ctypes.c_void_p * len(ps))(*[p.data_ptr() for p in ps])
    log_probs = torch.empty(B, T, CFG.vocab_padded, device="cuda")
    _lib.call(entry, ctypes.byref(model._native_model), _ptr(rows), B, T, pools(k_pools), pools(v_pools), _ptr(table), _ptr(cached),
              _ptr(total), _ptr(pos_start), table.size(1), k_pools[0].size(1), k_pools[0].size(0), _ptr(scales), _ptr(cnn_state), B,
              _ptr(slots), ctypes.c_void_p(scratch.data_ptr() + base), need, _ptr(log_probs), None,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert ob.device_status() == 0 and torch.isfinite(log_probs).all()
    sizes = [M * d * 4, M * d * 2, M * d * 2, M * CFG.ffn * 2, M * 4 * d * 2, M * d * 2]
    starts = base + np.cumsum([0] + [(s + 255) // 256 * 256 for s in sizes])
    take = lambda i: scratch[int(starts[i]):int(starts[i]) + sizes[i]].clone().view(rows.dtype)
    return take(4).view(B, T, 4 * d), take(5).view(B, T, d)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("block,pages,T", [(16, 64, 16), (16, 41, 5), (32, 33, 9), (32, 5, 16), (64, 6, 1), (128, 3, 16), (128, 34, 7), (16, 2, 16)])
def test_pages_and_attention_of_a_step(entry, dtype, fp8, block, pages, T):
    """Streams that begin a page, begin inside one, end inside one, fill the table, run past it, lie wholly past it, have no page
    for the chunk (dropped, never written) or see nothing.  Pages: bit for bit, all others untouched.  Attention: probabilities
    and outputs rounded once to 16 bits, fp32 sums, and with fp8 pages the scaled queries rounded to fp16."""
    H, d, D = CFG.heads, CFG.d_model, 64
    end = block * pages
    cached = [c for c in (0, 5, 31, 33, end // 2 + 3, end - T, end - 3) if 0 <= c] + [end, pages // 2 * block, 7]
    total = [c + T for c in cached]
    total[-2], total[-1] = cached[-2], 0
    B = len(cached)
    g = torch.Generator(device="cuda").manual_seed(block * 1000 + pages * 20 + T)
    model = ConformerCTC(ConformerConfig(**{f: getattr(CFG, f) for f in ConformerConfig.__dataclass_fields__}), OC.init_params(CFG, 77, 0.1),
                         dtype=dtype)
    model.forward_chunk_paged(torch.zeros(1, 67, 80, device="cuda"), [0], model.new_streaming_cache(1, 16))    # builds the position table
    num_blocks = B * pages + 2
    table = torch.randperm(num_blocks, generator=g, device="cuda")[:B * pages].view(B, pages).int()
    table[B - 2, cached[-2] // block:] = -1                          # no page for this stream's chunk
    at = torch.tensor(cached, dtype=torch.int32, device="cuda")
    seen = torch.tensor(total, dtype=torch.int32, device="cuda")
    pos_start = torch.randint(0, 900, (B,), generator=g, device="cuda", dtype=torch.int32)
    rows = torch.randn(B * T, model._native_model.embed_in, generator=g, device="cuda").to(dtype)
    cnn = torch.randn(CFG.layers, B, CFG.kernel - 1, d, generator=g, device="cuda").to(dtype)
    shape = (CFG.layers, num_blocks, block, H, D)
    scales = None
    if fp8:
        scales = torch.rand(CFG.layers, 2, H, generator=g, device="cuda") * 0.02 + 0.01
        k, v = (torch.randint(0, 0x70, shape, generator=g, device="cuda", dtype=torch.uint8) +
                128 * torch.randint(0, 2, shape, generator=g, device="cuda", dtype=torch.uint8) for _ in range(2))
    else:
        k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for _ in range(2))
    want_k, want_v = k[-1].clone(), v[-1].clone()
    qkv4, got = _step(entry, model, rows, B, T, list(k), list(v), table, at, seen, pos_start, scales, cnn)

    # the append
    fresh = qkv4.view(B, T, 4, H, D)
    for pool, new, which in ((want_k, fresh[:, :, 2], 0), (want_v, fresh[:, :, 3], 1)):
        if fp8:
            inv = (1.0 / scales[-1, which]).view(1, 1, H, 1)
            new = (new.float() * inv).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        for b in range(B):
            for t in range(T):
                col = (cached[b] + t) // block
                if col < pages and int(table[b, col]) >= 0:
                    pool[int(table[b, col]), (cached[b] + t) % block] = new[b, t]
    assert torch.equal(k[-1], want_k) and torch.equal(v[-1], want_v)

    # the attention
    def values(pool, which):
        return pool.view(torch.float8_e4m3fn).double() * scales[-1, which].double().view(1, 1, H, 1) if fp8 else pool.double()
    keys_all, vals_all = values(want_k, 0), values(want_v, 1)
    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -11      # of the output; of the probabilities too, fp16 with fp8 pages
    p_unit = 2.0 ** -11 if fp8 else unit
    pos = model._pos_proj[:, (CFG.layers - 1) * d:].double()
    for b in range(B):
        n = min(max(total[b], 0), end)
        if n == 0:
            assert torch.count_nonzero(got[b]) == 0
            continue
        where = (table[b].long().clamp(min=0)[:, None] * block + torch.arange(block, device="cuda")).reshape(-1)[:n]
        kk, vv = keys_all.view(-1, H, D)[where], vals_all.view(-1, H, D)[where]
        pp = torch.zeros(n, H, D, dtype=torch.double, device="cuda")
        have = pos[int(pos_start[b]):int(pos_start[b]) + n].view(-1, H, D)
        pp[:have.size(0)] = have
        qu, qv = fresh[b, :, 0].double(), fresh[b, :, 1].double()
        dot = lambda a, c: torch.einsum("qhd,khd->hqk", a, c)
        s = (dot(qu, kk) + dot(qv, pp)) * D ** -0.5
        out = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), vv)
        size = (dot(qu.abs(), kk.abs()) + dot(qv.abs(), pp.abs())).max().item() * D ** -0.5
        score = size * ((2.0 ** -11 if fp8 else 0.0) + 2 * D * 2.0 ** -24)
        bound = vv.abs().max() * (2 * p_unit + 2 * score + n * 2.0 ** -24) + unit * out.abs() + 1e-5
        err = (got[b].double().view(T, H, D) - out).abs()
        assert bool((err <= bound).all()), (b, cached[b], (err - bound).max().item(), err.max().item())


@pytest.mark.parametrize("entry", ENTRIES)
def test_append_positions_that_leave_32_bits_or_begin_below_zero(entry):
    """No row outside the table is written, and none inside it by a position that wrapped round."""
    block, pages, T, d = 16, 4, 16, CFG.d_model
    cached = [2 ** 31 - 5, 2 ** 31 - 1, -3, -2 ** 31]
    B = len(cached)
    g = torch.Generator(device="cuda").manual_seed(41)
    model = ConformerCTC(ConformerConfig(**{f: getattr(CFG, f) for f in ConformerConfig.__dataclass_fields__}), OC.init_params(CFG, 77, 0.1))
    model.forward_chunk_paged(torch.zeros(1, 67, 80, device="cuda"), [0], model.new_streaming_cache(1, 16))
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table = torch.randperm(B * pages, generator=g, device="cuda").view(B, pages).int()
    k, v = (torch.randn(CFG.layers, B * pages, block, CFG.heads, 64, generator=g, device="cuda").bfloat16() for _ in range(2))
    want_k, want_v = k[-1].clone(), v[-1].clone()
    qkv4, _ = _step(entry, model, torch.randn(B * T, model._native_model.embed_in, generator=g, device="cuda").bfloat16(), B, T, list(k), list(v),
                    table, ints(cached), ints([T] * B), ints([0] * B), None, torch.zeros(CFG.layers, B, CFG.kernel - 1, d, device="cuda").bfloat16())
    fresh = qkv4.view(B, T, 4, CFG.heads, 64)
    want_k[table[2, 0].long(), :T - 3], want_v[table[2, 0].long(), :T - 3] = fresh[2, 3:, 2], fresh[2, 3:, 3]
    assert torch.equal(k[-1], want_k) and torch.equal(v[-1], want_v)
