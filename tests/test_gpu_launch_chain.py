"""GPU: the executors' chained launches against weights that a kernel of this library wrote just before on the same stream."""
import pytest
import torch

import oasr_b200 as ob
from oasr_b200.encoder import ConformerConfig, ConformerCTC
from oasr_b200.fastconformer import FastConformerLayers
from oracle import conformer as OC
from oracle import fastconformer as OFC

pytestmark = pytest.mark.gpu


def _written_just_before(monkeypatch, entry, weight, value):
    """Right before the executor call ``entry``, on its stream and with no host wait, library kernels that let their successor
    start early write ``value`` into the model's ``weight``: a copy over many rows, then the row copy itself."""
    from oasr_b200 import _lib
    from oasr_b200.cache import gather_rows, scatter_rows

    plain = _lib.call
    index = torch.arange(value.size(0), device="cuda")
    ballast = torch.randn(1 << 16, 1024, device="cuda")
    back = torch.arange(ballast.size(0) - 1, -1, -1, device="cuda")

    def call(name, *args):
        if name == entry:
            monkeypatch.setattr(_lib, "call", plain)
            gather_rows(ballast, back)
            scatter_rows(weight, index, value)
        plain(name, *args)

    monkeypatch.setattr(_lib, "call", call)


def test_packed_batch_reads_weights_written_on_its_stream(monkeypatch):
    """4000 rows: the embedding runs on a kernel that triggers at once, the projection of the position table (few rows) on
    one that can fetch its weights early."""
    cfg = OC.TINY
    model = ConformerCTC(ConformerConfig(**{f: getattr(cfg, f) for f in ConformerConfig.__dataclass_fields__}), OC.init_params(cfg, 5, 0.1))
    feats, lengths = torch.randn(16, 1003, cfg.input_size, generator=torch.Generator().manual_seed(2)).cuda(), [1003] * 16
    want = model.forward_offline_packed(feats, lengths)[0].clone()
    value = model.pos_w_all.clone()
    for _ in range(4):
        model.pos_w_all.fill_(float("nan"))
        _written_just_before(monkeypatch, "oasr_b200_conformer_encode_packed", model.pos_w_all, value)
        got = model.forward_offline_packed(feats, lengths)[0]
        assert ob.device_status() == 0 and torch.equal(got, want)


def test_streaming_step_reads_weights_written_on_its_stream(monkeypatch):
    """1600 rows of a FastConformer step: the first Linear (4096 columns) runs on a kernel that triggers at once, the second one
    of the feed-forward (1024 columns) on one that can fetch its weights early."""
    cfg = OFC.FastConformerConfig(hidden=1024, heads=8, ffn=4096, layers=1, kernel=9, sliding_window=57, lookahead=3, bias=False)
    model = FastConformerLayers(cfg.hidden, cfg.heads, cfg.ffn, cfg.layers, cfg.kernel, cfg.sliding_window, cfg.lookahead,
                                OFC.init_params(cfg, 3, w_std=0.02))
    hidden = torch.randn(100, 16, cfg.hidden, generator=torch.Generator().manual_seed(2)).cuda()
    step = lambda: model.forward_chunk(hidden, list(range(100)), model.new_streaming_cache(100))
    want = step()
    weight = model.layers[0]["feed_forward1"][2]
    value = weight.clone()
    for _ in range(4):
        weight.fill_(float("nan"))
        _written_just_before(monkeypatch, "oasr_b200_fastconformer_chunk_paged", weight, value)
        got = step()
        assert ob.device_status() == 0 and torch.equal(got, want)
