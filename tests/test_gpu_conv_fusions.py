"""GPU: the FastConformer's fused conv steps against their separate operators and fp64."""
import pytest
import torch
import torch.nn.functional as F

from oasr_b200 import fused

pytestmark = pytest.mark.gpu

# relative error of a rounding to 16 bits (8 and 11 significant bits)
TOL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _conv_norm(x, w, b, nw, nb, dtype, eps=1e-5):
    """fp64: rows (8 + T, C) whose first 8 are the history -> (T, C), and what the conv's rounding may add to the error."""
    x, w, b, nw, nb = (t.double().cpu() for t in (x, w, b, nw, nb))
    y = F.conv1d(x.t()[None], w.t()[:, None], b, groups=x.size(1))[0].t()
    # what the rounding of a conv value (TOL, relative) can move its output by: SiLU's slope is at most 1.1
    slack = 1.1 * TOL[dtype] * y.abs() / (y.var(1, unbiased=False, keepdim=True) + eps).sqrt() * nw.abs()
    return F.silu(F.layer_norm(y, (x.size(1),), nw, nb, eps)), slack


def _params(C, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g)
    return [t.to(dtype).cuda() for t in (r(9, C) * 0.3, r(C) * 0.1, 1 + 0.1 * r(C), 0.1 * r(C))], g


def _check(got, want, dtype):
    # beside the two roundings: what those of the other channels move the mean and the variance by (a tenth of the conv's own
    # rounding and 0.05 of a unit), and fp32 sums
    want, slack = want
    err = (got.double().cpu() - want).abs()
    assert bool((err <= TOL[dtype] * (want.abs() + 0.05) + 1.1 * slack).all()), err.max().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C,lens", [(1024, [1, 7, 8, 9, 31, 32, 33, 100]), (128, [40, 3]), (384, [17]), (512, [150] * 70), (1024, [40] * 150)])
def test_packed_depthwise_conv_norm_swish(dtype, C, lens):
    (w, b, nw, nb), g = _params(C, dtype, C)
    x = torch.randn(sum(lens), C, generator=g).to(dtype).cuda()
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    got = fused.dwconv_norm_swish_packed(x, w, b, nw, nb, cu, max(lens))
    at = 0
    for n in lens[:8]:
        _check(got[at:at + n], _conv_norm(torch.cat([x.new_zeros(8, C), x[at:at + n]]), w, b, nw, nb, dtype), dtype)
        at += n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [1, 4, 8, 9, 16, 17])
def test_streaming_depthwise_conv_norm_swish(dtype, T):
    C, slots = 256, [5, 0, 3, 99]                     # 99: outside the buffer, an empty left context that is not kept
    (w, b, nw, nb), g = _params(C, dtype, T)
    state = torch.randn(6, 8, C, generator=g).to(dtype).cuda()
    x = torch.randn(len(slots), T, C, generator=g).to(dtype).cuda()
    before = state.clone()
    got = fused.dwconv_norm_swish_stream(x, w, b, nw, nb, state, torch.tensor(slots, dtype=torch.int64).cuda())
    for i, slot in enumerate(slots):
        rows = torch.cat([before[slot] if slot < 6 else x.new_zeros(8, C), x[i]])
        _check(got[i], _conv_norm(rows, w, b, nw, nb, dtype), dtype)
        if slot < 6:
            before[slot] = rows[-8:]
    assert torch.equal(state, before)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,Fb,C,lens", [(1, 3, 128, 256, [3]), (3, 41, 80, 256, [41, 17, 1]), (2, 64, 7, 128, [64, 9]),
                                           (40, 130, 128, 256, list(range(91, 131))), (2, 30, 1, 512, [30, 5])])
def test_stem_and_depthwise_conv_in_one(dtype, B, T, Fb, C, lens):
    assert fused.subsample_stem_dw_supported(Fb, C)
    g = torch.Generator().manual_seed(T + C)
    feats = torch.randn(B, T, Fb, generator=g).cuda()
    w1, b1 = torch.randn(C, 3, 3, generator=g).cuda() * 0.5, torch.randn(C, generator=g).cuda() * 0.1
    w2, b2 = (torch.randn(C, 3, 3, generator=g) * 0.5).to(dtype).cuda(), (torch.randn(C, generator=g) * 0.1).to(dtype).cuda()
    mid = torch.tensor([n // 2 + 1 for n in lens], dtype=torch.int32).cuda()
    out = mid // 2 + 1
    x = fused.subsample_conv1(F.pad(feats, (2, 1, 2, 1)), w1, b1, dtype, t1_limit=mid)
    want = fused.depthwise_conv2d_k3s2(x, w2, b2, 2, 1, out_len=out, in_len=mid)
    got = fused.subsample_stem_dw(feats, w1, b1, w2, b2, mid, out)
    assert got.shape == want.shape and torch.equal(got, want)


# (SL + T) * slab pieces of a block: one, two and four per thread, narrower slabs, the last size of the kernel and the first of
# the two launches behind it; inputs shorter than the state
@pytest.mark.parametrize("SL,T,C,dtype", [(8, 16, 256, torch.bfloat16), (14, 3, 72, torch.float16), (2, 40, 80, torch.float32),
                                          (14, 100, 64, torch.bfloat16), (2, 300, 24, torch.float32), (2, 1022, 8, torch.bfloat16),
                                          (2, 1023, 72, torch.bfloat16), (0, 5, 8, torch.float16)])
def test_conv_state_is_concatenated_and_rolled(SL, T, C, dtype):
    from oasr_b200 import _lib
    from oasr_b200.functional import _DTYPE_ID

    g = torch.Generator().manual_seed(SL + T)
    state, x = torch.randn(5, SL, C, generator=g).to(dtype).cuda(), torch.randn(4, T, C, generator=g).to(dtype).cuda()
    slots = [3, -1, 0, 7]                                   # two outside the buffer: zeros before the input, nothing kept
    want_state = state.clone()
    before = [state[s] if 0 <= s < 5 else torch.zeros_like(state[0]) for s in slots]
    want = torch.stack([torch.cat([b, x[i]]) for i, b in enumerate(before)])
    for i, s in enumerate(slots):
        if 0 <= s < 5:
            want_state[s] = want[i, T:]
    got, ids = torch.full_like(want, 7.0), torch.tensor(slots).cuda()
    held = state if SL else torch.empty(5, 1, C, dtype=dtype, device="cuda")       # an empty tensor has no address
    _lib.call("oasr_b200_conv_state_concat", got.data_ptr(), held.data_ptr(), 5, ids.data_ptr(), x.data_ptr(), 4, SL, T, C,
              _DTYPE_ID[dtype], torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, want) and torch.equal(state, want_state)


def test_other_kernel_sizes_keep_the_separate_steps():
    """A conv of 5 taps: packed batches native and composed agree bit for bit, streams continue their cached tail (chunks
    against the offline pass, tolerance of the streaming tests: the two attend through different kernels in bf16)."""
    from oasr_b200.fastconformer import FastConformerLayers
    from oracle import fastconformer as OFC

    cfg = OFC.FastConformerConfig(hidden=256, heads=2, ffn=512, layers=2, kernel=5, sliding_window=25, lookahead=3, bias=True)
    model = FastConformerLayers(cfg.hidden, cfg.heads, cfg.ffn, cfg.layers, cfg.kernel, cfg.sliding_window, cfg.lookahead,
                                OFC.init_params(cfg, 21))
    assert not fused.dwconv_norm_swish_supported(cfg.hidden, cfg.kernel)
    lengths, hidden = [64, 17, 1], torch.randn(3, 64, 256, generator=torch.Generator().manual_seed(4)).cuda()
    native, _ = model.forward_rows(hidden, lengths)
    model.native = False
    composed, _ = model.forward_rows(hidden, lengths)
    model.native = True
    assert torch.equal(native, composed)
    cache = model.new_streaming_cache(max_streams=3, chunk_frames=16)
    chunks = torch.cat([model.forward_chunk(hidden[:1, 16 * c:16 * (c + 1)], [2], cache) for c in range(4)], 1)
    d = (chunks[0] - model.forward(hidden[:1], [64])[0]).abs()
    assert d.max().item() < 6e-2 and d.mean().item() < 6e-3
