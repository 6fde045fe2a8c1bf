"""GPU parity: norm / activation / depthwise-conv kernels vs the CPU oracle.

Cases follow the reference's kernel unit tests (tests/test_norm.py,
tests/test_activation.py, tests/test_conv.py): same shapes families, same
tolerances or tighter, plus ragged / empty / non-vectorisable extents.
"""
import numpy as np
import pytest
import torch

import oasr_b200 as ob
from oracle import ops as O

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16, torch.float32]
TOL = {torch.bfloat16: 2e-2, torch.float16: 3e-3, torch.float32: 2e-5}


def _rand(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype)


def _close(got, want, dtype, scale=1.0):
    got = got.float().cpu()
    want = want.float()
    # the oracle's fp32 result rounded to the kernel's output type is the target
    want_r = want.to(dtype).float()
    tol = TOL[dtype] * scale
    err = (got - want_r).abs().max().item() if got.numel() else 0.0
    assert err <= tol * max(1.0, want.abs().max().item() if want.numel() else 1.0), f"max err {err}"


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(4, 250, 512), (3, 7, 256), (2, 5, 1024), (1, 1, 8), (2, 3, 80), (5, 333),
                                   (2, 4, 4096), (2, 4, 4104), (0, 16), (3, 5, 12)])
def test_layer_norm(dtype, shape):
    x = _rand(shape, dtype, 1, 2.0)
    H = shape[-1]
    w, b = _rand((H,), dtype, 2) + 1, _rand((H,), dtype, 3)
    got = ob.layer_norm(x.cuda(), w.cuda(), b.cuda(), 1e-5)
    _close(got, O.layer_norm(x, w, b, 1e-5), dtype)
    got = ob.layer_norm(x.cuda(), w.cuda(), None, 1e-5)
    _close(got, O.layer_norm(x, w, None, 1e-5), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("act", [0, 1, 2, 4])
def test_layer_norm_activation(dtype, act):
    x = _rand((3, 17, 512), dtype, 4)
    w, b = _rand((512,), dtype, 5) + 1, _rand((512,), dtype, 6)
    got = ob.layer_norm_activation(x.cuda(), w.cuda(), b.cuda(), 1e-5, act)
    _close(got, O.layer_norm(x, w, b, 1e-5, act), dtype)
    got = ob.rms_norm_activation(x.cuda(), w.cuda(), b.cuda(), 1e-5, act)
    _close(got, O.rms_norm(x, w, b, 1e-5, act), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(4, 250, 512), (2, 3, 1000), (7, 24)])
def test_rms_norm(dtype, shape):
    x = _rand(shape, dtype, 7, 3.0)
    H = shape[-1]
    w, b = _rand((H,), dtype, 8) + 1, _rand((H,), dtype, 9)
    _close(ob.rms_norm(x.cuda(), w.cuda(), None, 1e-5), O.rms_norm(x, w, None, 1e-5), dtype)
    _close(ob.rms_norm(x.cuda(), w.cuda(), b.cuda(), 1e-6), O.rms_norm(x, w, b, 1e-6), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(4, 250, 512), (2, 9, 256), (3, 5, 12)])
@pytest.mark.parametrize("alpha", [1.0, 0.5])
def test_add_layer_norm_residual(dtype, shape, alpha):
    x, r = _rand(shape, dtype, 10), _rand(shape, dtype, 11, 2.0)
    H = shape[-1]
    w, b = _rand((H,), dtype, 12) + 1, _rand((H,), dtype, 13)
    out, res = ob.add_layer_norm_residual(x.cuda(), r.cuda(), w.cuda(), b.cuda(), 1e-5, alpha)
    want_out, want_res = O.add_layer_norm_residual(x, r, w, b, 1e-5, alpha)
    _close(out, want_out, dtype)
    # the carried sum is the fp32 sum rounded ONCE: bit-exact (reference tests/test_norm.py:276-281)
    want_fma = torch.addcmul(r.float(), torch.tensor(alpha), x.float()).to(dtype)
    assert torch.equal(res.cpu(), want_res) or torch.equal(res.cpu(), want_fma)
    out2 = ob.add_layer_norm(x.cuda(), r.cuda(), w.cuda(), b.cuda(), 1e-5, alpha=alpha)
    assert torch.equal(out2, out)
    o3, r3 = ob.add_rms_norm_residual(x.cuda(), r.cuda(), w.cuda(), b.cuda(), 1e-5, alpha)
    w_o3, w_r3 = O.add_rms_norm_residual(x, r, w, b, 1e-5, alpha)
    _close(o3, w_o3, dtype)
    assert torch.equal(r3.cpu(), w_r3) or torch.equal(r3.cpu(), want_fma)
    assert torch.equal(ob.add_rms_norm(x.cuda(), r.cuda(), w.cuda(), b.cuda(), 1e-5, alpha), o3)


def test_norm_rejects_padded_rows_and_cpu():
    x = torch.randn(4, 8, 64, device="cuda", dtype=torch.bfloat16)[:, :, :32]
    w = torch.ones(32, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        ob.layer_norm(x, w)
    with pytest.raises(RuntimeError):
        ob.layer_norm(torch.randn(2, 32), torch.ones(32))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(4, 250, 512), (2, 7, 256), (3, 5, 20), (1, 3, 1024)])
@pytest.mark.parametrize("act", [-1, 2, 0])
def test_batch_norm(dtype, shape, act):
    x = _rand(shape, dtype, 14, 2.0)
    C = shape[-1]
    w, b = _rand((C,), dtype, 15) + 1, _rand((C,), dtype, 16)
    mean, var = _rand((C,), dtype, 17), _rand((C,), dtype, 18).abs() + 0.5
    want = O.batch_norm(x, w, b, mean, var, 1e-5, act)
    args = [t.cuda() for t in (x, w, b, mean, var)]
    if act == -1:
        got = ob.batch_norm_1d(*args, 1e-5)
    elif act == 2:
        got = ob.batch_norm_swish(*args, 1e-5)
    else:
        got = ob.batch_norm_activation(*args, 1e-5, act)
    _close(got, want, dtype, scale=2.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(4, 250, 1024), (2, 3, 16), (3, 5, 24), (1, 1, 2), (0, 4, 64)])
def test_glu_swish(dtype, shape):
    x = _rand(shape, dtype, 19, 2.0)
    _close(ob.glu(x.cuda()), O.glu(x), dtype)
    _close(ob.swish(x.cuda()), O.swish(x), dtype)
    out = torch.empty_like(x, device="cuda")
    assert ob.swish(x.cuda(), out=out) is out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("B,T,C,K,pad", [(4, 250, 256, 15, 7), (2, 100, 512, 15, (14, 0)), (3, 33, 64, 9, (8, 0)),
                                          (1, 30, 512, 15, 0), (2, 17, 24, 3, 1), (2, 40, 10, 4, (2, 1)),
                                          (1, 5, 64, 15, 7), (2, 64, 128, 31, 15)])
def test_depthwise_conv1d(dtype, B, T, C, K, pad):
    x = _rand((B, T, C), dtype, 20)
    w = _rand((K, 1, C), dtype, 21, 0.3)
    b = _rand((C,), dtype, 22)
    got = ob.depthwise_conv1d(x.cuda(), w.cuda(), b.cuda(), pad)
    _close(got, O.depthwise_conv1d(x, w, b, pad), dtype, scale=2.0)
    got = ob.depthwise_conv1d(x.cuda(), w.cuda().reshape(K, C), None, pad)
    _close(got, O.depthwise_conv1d(x, w, None, pad), dtype, scale=2.0)
    got = ob.depthwise_conv1d_silu(x.cuda(), w.cuda(), b.cuda(), pad)
    _close(got, O.depthwise_conv1d(x, w, b, pad, act=2), dtype, scale=2.0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bool_mask", [True, False])
def test_depthwise_conv1d_fsmn_mask(dtype, bool_mask):
    B, T, C, K = 3, 40, 64, 11
    x = _rand((B, T, C), dtype, 23)
    w = _rand((K, C), dtype, 24, 0.3)
    lens = torch.tensor([40, 25, 1])
    mask = (torch.arange(T)[None, :] < lens[:, None]).unsqueeze(-1)
    m = mask if bool_mask else mask.to(dtype)
    got = ob.depthwise_conv1d(x.cuda(), w.cuda(), None, (K - 1) // 2, mask=m.cuda(), add_input=True)
    _close(got, O.depthwise_conv1d(x, w, None, (K - 1) // 2, mask=mask, add_input=True), dtype, scale=2.0)


# 16-bit types at kernel sizes 9 and 15: the rolling kernel takes the bool mask; T around its runs of 4 K frames
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K,T,C", [(9, 36, 64), (9, 73, 10), (15, 60, 256), (15, 7, 24), (15, 121, 514)])
@pytest.mark.parametrize("masked,add_input", [(True, False), (True, True), (False, True)])
def test_depthwise_conv1d_mask_of_the_rolling_kernel(dtype, K, T, C, masked, add_input):
    x, w, b = _rand((3, T, C), dtype, 33), _rand((K, C), dtype, 34, 0.3), _rand((C,), dtype, 35)
    mask = (torch.arange(T)[None, :] < torch.tensor([T, (T + 1) // 2, 1])[:, None]).unsqueeze(-1) if masked else None
    if masked:          # padding that is no number: the input is multiplied by the mask, here as everywhere
        x[1, -1, :2], x[2, -1, 2:4] = float("inf"), float("nan")
        x[1, -2, 4:6] = -torch.finfo(dtype).max
    got = ob.depthwise_conv1d(x.cuda(), w.cuda(), b.cuda(), (K - 1) // 2, mask=mask.cuda() if masked else None, add_input=add_input)
    want = O.depthwise_conv1d(x, w, b, (K - 1) // 2, mask=mask, add_input=add_input)
    # one rounding (half an ulp, 2^-9 / 2^-12 of the value) and K + 1 fp32 additions of values of a few units
    torch.testing.assert_close(got.float().cpu(), want, rtol=2.0 ** (-8 if dtype == torch.bfloat16 else -11), atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("K", [9, 11, 15])
def test_masked_depthwise_conv1d_swish_is_exact_to_the_rounding(K):
    """The C entry point takes a mask together with swish: half an ulp of fp16 from the exact value, whichever kernel runs
    (a swish by one tanh.approx, relative error 2^-11, is not)."""
    from oasr_b200 import _lib

    B, T, C = 2, 90, 64
    x, w, b = _rand((B, T, C), torch.float16, 41), _rand((K, C), torch.float16, 42, 0.3), _rand((C,), torch.float16, 43)
    mask = torch.arange(T)[None, :] < torch.tensor([T, 50])[:, None]
    out = torch.empty(B, T, C, dtype=torch.float16, device="cuda")
    dev = [t.cuda() for t in (x, w, b, mask)]
    _lib.call("oasr_b200_depthwise_conv1d", out.data_ptr(), *(t.data_ptr() for t in dev[:3]), B, T, C, K, (K - 1) // 2, (K - 1) // 2,
              dev[3].data_ptr(), 1, 0, 2, 1, torch.cuda.current_stream().cuda_stream)
    m = mask[..., None].double()
    y = torch.nn.functional.conv1d((x.double() * m).transpose(1, 2), w.double().t()[:, None], b.double(), padding=(K - 1) // 2,
                                   groups=C).transpose(1, 2) * m
    y = torch.nn.functional.silu(y)
    half_ulp = torch.ldexp(torch.ones_like(y), torch.frexp(y)[1].clamp(min=-13) - 12)
    # beside it: K + 1 fp32 additions and an exponential of 2 ulp on values of a few units, 16 * 2^-24 each
    assert ((out.double().cpu() - y).abs() <= half_ulp + 1e-6 * (1 + y.abs())).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [16, 3, 1])
def test_causal_conv1d_state(dtype, T):
    B, C, K = 3, 64, 9
    w = _rand((C, 1, K), dtype, 25, 0.3)
    b = _rand((C,), dtype, 26)
    state = _rand((B, K - 1, C), dtype, 27)
    st_gpu = state.cuda().clone()
    for step in range(3):
        x = _rand((B, T, C), dtype, 28 + step)
        want, state = O.causal_conv1d(x, state, w, b)
        got = ob.causal_conv1d(x.cuda(), st_gpu, w.cuda(), b.cuda())
        _close(got, want, dtype, scale=2.0)
        assert torch.equal(st_gpu.cpu(), state)  # rolled state is a pure copy: bit-exact


@pytest.mark.parametrize("conv1_mma", [1, 0])
@pytest.mark.parametrize("C,lens", [(128, [96, 151, 40]), (512, [403, 67, 1000, 250]), (256, [67] * 5)])
def test_subsampling_front_end_matches_torch_conv2d(C, lens, conv1_mma):
    """conv1 (parity-split layout: split-bf16 GEMM on the tensor cores for 256 / 512 channels, else - or with the
    tunable off - the fp32 stencil) + conv2 (tcgen05 implicit GEMM, packed valid frames) against torch conv2d + ReLU
    in fp32 on the same 16-bit-rounded weights and intermediate."""
    from oasr_b200 import fused, tunables

    tunables.set("conv1_mma", conv1_mma)
    try:
        _front_end_case(C, lens, stencil=not (conv1_mma and C in (256, 512)))
    finally:
        tunables.set("conv1_mma", 1)


def _front_end_case(C, lens, stencil):
    from oasr_b200 import fused

    torch.manual_seed(5)
    B, T, F = len(lens), max(lens), 80
    feats = torch.randn(B, T, F, device="cuda")
    w1 = torch.randn(C, 3, 3, device="cuda") * 0.3
    b1 = torch.randn(C, device="cuda") * 0.1
    w2 = (torch.randn(C, 3, 3, C, device="cuda") * (9 * C) ** -0.5).bfloat16()
    b2 = (torch.randn(C, device="cuda") * 0.1).bfloat16()
    out_lens = [(n - 3) // 4 for n in lens]
    cu = torch.tensor([0] + list(np.cumsum(out_lens)), dtype=torch.int32, device="cuda")
    total = int(cu[-1])
    t1_limit = torch.tensor([2 * n + 1 for n in out_lens], dtype=torch.int32, device="cuda")
    T1, F1 = (T - 3) // 2 + 1, (F - 3) // 2 + 1
    x1 = fused.subsample_conv1_s2d(feats, w1, b1, torch.bfloat16, t1_limit=t1_limit)
    got = fused.subsample_conv2(x1, T1, F1, w2, b2, cu, total).float()
    assert ob.device_status() == 0
    # reference
    y1_f32 = torch.relu(torch.nn.functional.conv2d(feats[:, None], w1[:, None], b1, stride=2))                  # (B,C,T1,F1)
    y1 = y1_f32.bfloat16().float()
    # conv1 against the NHWC kernel and the parity-split layout
    nhwc = fused.subsample_conv1(feats, w1, b1, torch.bfloat16).float()
    assert (nhwc - y1.permute(0, 2, 3, 1)).abs().max().item() < 2e-2
    for b, n in enumerate(out_lens):
        lim = 2 * n + 1
        t1 = torch.arange(lim, device="cuda")
        f1 = torch.arange(F1, device="cuda")
        plane = (t1[:, None] & 1) * 2 + (f1[None] & 1)
        s2d = x1[b][t1[:, None] // 2, plane, f1[None] // 2].float()             # (lim, F1, C)
        if stencil:
            assert torch.equal(s2d, nhwc[b, :lim])
        else:
            # products of two-term bf16 operands (the lo x lo term dropped: 2^-16 of the summed magnitudes), one rounding
            # on store: within one 16-bit rounding step of the exact value plus that share of sum |x||w| + |b|
            # everywhere, and the same 16-bit value as the fp32 stencil almost everywhere
            exact = y1_f32[b, :, :lim].permute(1, 2, 0)
            mag = torch.nn.functional.conv2d(feats[b:b + 1, None].abs(), w1[:, None].abs(), b1.abs(), stride=2)[0, :, :lim].permute(1, 2, 0)
            assert ((s2d - exact).abs() <= exact.abs() * 2.0 ** -8 + mag * 2.0 ** -14 + 1e-6).all()
            assert (s2d != nhwc[b, :lim]).float().mean().item() < 2e-3
    y2 = torch.relu(torch.nn.functional.conv2d(y1, w2.float().permute(0, 3, 1, 2), b2.float(), stride=2))      # (B,C,T2,F2)
    want = torch.cat([y2[b, :, :n].permute(1, 2, 0).reshape(n, -1) for b, n in enumerate(out_lens)])
    err = (got - want).abs().max().item()
    assert err < 3e-2, err


@pytest.mark.parametrize("K,causal", [(15, False), (9, True)])
def test_packed_depthwise_conv_kernels_agree_with_each_other_and_with_fp32(K, causal):
    """The rolling register-window kernel (default for kernel sizes 9 / 15) against the run-at-once kernel
    (``dwconv_path`` 0) and an fp32 torch restatement, on ragged segments incl. ones shorter than the kernel, a run
    boundary inside a segment (60 frames), folded BatchNorm + swish (non-causal form) and the padded-semantics fill."""
    from oasr_b200 import fused, tunables

    torch.manual_seed(11)
    lens = [1, 7, 59, 60, 61, 120, 121, 333, 14, 15]
    C = 512
    total = sum(lens)
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32).cuda()
    x = torch.randn(total, C).bfloat16().cuda()
    w = (torch.randn(K, C) * 0.3).bfloat16().cuda()
    b = torch.randn(C).bfloat16().cuda()
    sc, sh = (torch.rand(C) + 0.5).cuda(), torch.randn(C).cuda()
    fill = torch.randn(C).cuda()
    fill_frames = torch.tensor([min((K - 1) // 2, 3 + i % 5) for i in range(len(lens))], dtype=torch.int32).cuda()

    def run():
        if causal:
            return fused.depthwise_conv1d_packed_causal(x, w, b, cu, max(lens), activation=-1).float()
        return fused.depthwise_conv1d_packed(x, w, b, cu, max(lens), post_scale=sc, post_shift=sh, right_fill=fill,
                                             fill_frames=fill_frames, activation=2).float()

    outs = {}
    for path in (2, 0):
        tunables.set("dwconv_path", path)
        try:
            outs[path] = run()
        finally:
            tunables.set("dwconv_path", 2)
    assert ob.device_status() == 0
    assert (outs[2] - outs[0]).abs().max().item() < 4e-2      # two roundings to bf16 of nearly equal fp32 values
    xf, wf = x.float().cpu(), w.float().cpu()
    for s, n in enumerate(lens):
        a = int(cu[s])
        seg = xf[a:a + n]
        if causal:
            padded = torch.cat([torch.zeros(K - 1, C), seg])
        else:
            nf = int(fill_frames[s])
            right = torch.cat([fill.cpu().bfloat16().float().expand(nf, C), torch.zeros((K - 1) // 2 - nf, C)])
            padded = torch.cat([torch.zeros((K - 1) // 2, C), seg, right])
        want = sum(padded[k:k + n] * wf[k] for k in range(K)) + b.float().cpu()
        if not causal:
            want = want * sc.cpu() + sh.cpu()
            want = want * torch.sigmoid(want)
        for path in (2, 0):
            err = (outs[path][a:a + n].cpu() - want).abs().max().item()
            assert err < 3e-2 * max(1.0, want.abs().max().item()), (path, s, n, err)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C,N,frames", [(512, 512, [1]), (512, 512, [6]), (512, 512, [7, 0, 5]), (512, 512, [102]), (512, 512, [108]), (512, 512, [216]),
                                        (512, 512, [438]), (512, 512, [444]), (512, 512, [16] * 12), (64, 256, [13, 40]), (128, 128, [9, 1, 3]),
                                        (64, 256, [7, 0, 1] * 11), (64, 512, [0] * 31 + [6] + [0] * 33 + [20, 3])])
def test_subsampling_second_conv_at_every_tile_width(C, N, frames, dtype):
    """Few tiles deal their output columns to several pairs of SMs: every width, the last sizes before each line and partial
    tiles; more utterances than lanes look for a tile at a time, empty ones among them; against fp64.  Bound: one rounding to 16 bits of the result and K fp32 additions of the products."""
    from oasr_b200 import fused

    g = torch.Generator(device="cuda").manual_seed(sum(frames) + C)
    F1, F2, B = 39, 19, len(frames)
    T1 = 2 * max(frames) + 1
    x = torch.randn(B, T1, F1, C, generator=g, device="cuda").to(dtype)
    w = (torch.randn(N, 3, 3, C, generator=g, device="cuda") * (9 * C) ** -0.5).to(dtype)
    b = (torch.randn(N, generator=g, device="cuda") * 0.1).to(dtype)
    split = torch.zeros(B, (T1 + 1) // 2, 4, (F1 + 1) // 2, C, dtype=dtype, device="cuda")
    for plane in range(4):
        part = x[:, plane >> 1::2, plane & 1::2]
        split[:, :part.size(1), plane, :part.size(2)] = part
    cu = torch.tensor([0] + list(np.cumsum(frames)), dtype=torch.int32, device="cuda")
    got = fused.subsample_conv2(split, T1, F1, w, b, cu, sum(frames)).view(-1, F2, N).double()
    assert ob.device_status() == 0
    at = 0
    for i, n in enumerate(frames):
        want = b.double().expand(n, F2, N).clone()
        size = b.double().abs().expand(n, F2, N).clone()
        for kh in range(3):
            for kw in range(3):
                rows = x[i, kh:kh + 2 * n - 1:2, kw:kw + 2 * F2 - 1:2].double() if n else x[i, :0, :F2].double()
                want += rows @ w[:, kh, kw].double().t()
                size += rows.abs() @ w[:, kh, kw].double().abs().t()
        want = want.relu()
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        bound = eps * want.abs() + 9 * C * 2.0 ** -24 * size
        assert bool(((got[at:at + n] - want).abs() <= bound).all()), (i, ((got[at:at + n] - want).abs() - bound).max().item())
        at += n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C,N", [(64, 128), (64, 256), (512, 512)])
def test_subsampling_second_conv_gives_an_utterance_the_same_bits_in_every_batch(C, N, dtype):
    """A batch's size chooses the columns of a tile, 64 to N; the first utterances' rows are those of each of them alone."""
    from oasr_b200 import fused

    g = torch.Generator(device="cuda").manual_seed(N)
    F1, F2, n, most = 39, 19, 6, 96
    T1 = 2 * n + 1
    x = torch.randn(most, (T1 + 1) // 2, 4, (F1 + 1) // 2, C, generator=g, device="cuda").to(dtype)      # parity planes
    w = (torch.randn(N, 3, 3, C, generator=g, device="cuda") * (9 * C) ** -0.5).to(dtype)
    b = (torch.randn(N, generator=g, device="cuda") * 0.1).to(dtype)

    def conv(utts):
        cu = torch.arange(0, (utts + 1) * n, n, dtype=torch.int32, device="cuda")
        return fused.subsample_conv2(x[:utts].contiguous(), T1, F1, w, b, cu, utts * n).clone()

    want = conv(most)
    assert ob.device_status() == 0 and torch.isfinite(want).all()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for utts in (1, sms // 16, sms // 16 + 1, sms // 8, sms // 8 + 1, sms // 4, sms // 4 + 1, most - 1):
        got = conv(utts)
        assert torch.equal(got, want[:got.size(0)]), utts
