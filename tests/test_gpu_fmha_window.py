"""GPU: windowed relative-position attention (packed segments, paged streams) against fp32 torch on the same operands."""
import pytest
import torch

import oasr_b200 as ob
from oasr_b200 import _lib, fused
from oasr_b200.functional import _DTYPE_ID, _p, _stream

pytestmark = pytest.mark.gpu


def _reference(qu, qv, k, v, rel, center, q_abs, k_abs, chunk, left_chunks, scale):
    """fp32, one segment: (n, H, D) queries at frames q_abs, (m, H, D) keys at frames k_abs."""
    qu, qv, k, v, rel = (t.float() for t in (qu, qv, k, v, rel))
    d = q_abs[:, None] - k_abs[None, :]
    r = rel[(center - d).clamp(0, rel.size(0) - 1)]                                    # (n, m, H, D)
    s = (torch.einsum("nhd,mhd->hnm", qu, k) + torch.einsum("nhd,nmhd->hnm", qv, r)) * scale
    diff = q_abs[:, None] // chunk - k_abs[None, :] // chunk
    s = s.masked_fill(~((diff >= 0) & (diff <= left_chunks))[None], float("-inf"))
    return torch.einsum("hnm,mhd->nhd", s.softmax(-1), v)


def _operands(rows, H, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, 4 * H * D, generator=g).to(dtype).cuda(), (torch.randn(64, H * D, generator=g) * 0.5).to(dtype).cuda()


# P and the output are rounded once: 2^-9 (bf16), 2^-12 (fp16) of values of a few units
TOL = {torch.bfloat16: 2e-2, torch.float16: 3e-3}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,chunk,left_chunks", [(128, 4, 14), (64, 4, 14), (128, 1, 0), (128, 3, 8), (64, 32, 0), (128, 16, 2), (128, 1, 62)])
def test_packed_segments(dtype, D, chunk, left_chunks):
    H, lens = 2, [1, 200, 5, 64, 65, 130, 16]
    assert fused.fmha_window_supported(D, chunk, left_chunks)
    qkv4, rel = _operands(sum(lens), H, D, dtype, D + chunk)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    center = left_chunks * chunk + chunk - 1
    out = fused.fmha_window_packed(qkv4, rel, center, cu, max(lens), H, chunk, left_chunks, D ** -0.5)
    assert ob.device_status() == 0
    at = 0
    for n in lens:
        qu, qv, k, v = qkv4[at:at + n].view(n, 4, H, D).unbind(1)
        frames = torch.arange(n, device="cuda")
        want = _reference(qu, qv, k, v, rel.view(64, H, D), center, frames, frames, chunk, left_chunks, D ** -0.5)
        assert (out[at:at + n].view(n, H, D).float() - want).abs().max().item() < TOL[dtype]
        at += n


def test_windows_that_do_not_fit_are_refused():
    assert not fused.fmha_window_supported(128, 4, 15) and not fused.fmha_window_supported(96, 4, 2) and not fused.fmha_window_supported(64, 33, 0)
    qkv4, rel = _operands(8, 2, 64, torch.bfloat16, 1)
    with pytest.raises(_lib.OasrB200Error, match="window"):
        fused.fmha_window_packed(qkv4, rel, 63, torch.tensor([0, 8], dtype=torch.int32).cuda(), 8, 2, 4, 15, 0.125)


@pytest.mark.parametrize("D,H,Tq,chunk,left_chunks", [(128, 8, 16, 4, 14), (64, 3, 24, 4, 6), (128, 2, 40, 2, 20)])
def test_paged_streams_write_their_pages_and_attend(D, H, Tq, chunk, left_chunks):
    """Streams with an empty, a part and a full history; the kernel's page writes against the oracle rule of write_kv_chunk."""
    dtype, bs, nblk, B = torch.bfloat16, 8, 16, 3
    cached = torch.tensor([0, 24, 64], dtype=torch.int32)
    pos_start = torch.tensor([0, 0, 32], dtype=torch.int32)
    g = torch.Generator().manual_seed(3)
    table = torch.randperm(B * nblk, generator=g).view(B, nblk).to(torch.int32).cuda()
    kp, vp = (torch.randn(B * nblk, bs, H, D, generator=g).to(dtype).cuda() for _ in range(2))
    qkv4, rel = _operands(B * Tq, H, D, dtype, 9)
    k_new, v_new = (qkv4.view(B, Tq, 4, H, D)[:, :, i].permute(0, 2, 1, 3) for i in (2, 3))
    want_k, want_v = kp.clone(), vp.clone()
    ob.write_kv_chunk(want_k, want_v, table, k_new, v_new, cached.cuda())
    out = torch.empty(B * Tq, H * D, dtype=dtype, device="cuda")
    cached_d, start_d = cached.cuda(), pos_start.cuda()
    center = left_chunks * chunk + chunk - 1
    _lib.call("oasr_b200_fmha_window_paged", _p(out), _p(qkv4), _p(kp), _p(vp), _p(rel), 64, center, _p(table), _p(cached_d), _p(start_d), B,
              Tq, H, D, nblk, bs, B * nblk, chunk, left_chunks, D ** -0.5, _DTYPE_ID[dtype], _stream(out))
    assert ob.device_status() == 0
    assert torch.equal(kp, want_k) and torch.equal(vp, want_v)
    for b in range(B):
        n = int(cached[b]) + Tq
        k, v = (pool[table[b].long()].reshape(nblk * bs, H, D)[:n] for pool in (kp, vp))
        qu, qv = qkv4.view(B, Tq, 4, H, D)[b, :, :2].unbind(1)
        frames = int(pos_start[b]) + torch.arange(n, device="cuda")
        want = _reference(qu, qv, k, v, rel.view(64, H, D), center, frames[int(cached[b]):], frames, chunk, left_chunks, D ** -0.5)
        assert (out.view(B, Tq, H, D)[b].float() - want).abs().max().item() < TOL[dtype]
