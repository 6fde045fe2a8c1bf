"""What the native streaming step refuses before it launches anything (no GPU: no address here is ever read)."""
import ctypes

import pytest

from oasr_b200 import _lib

BASE = 1 << 20                       # stands for a device buffer


@pytest.mark.parametrize("entry", ["oasr_b200_conformer_chunk_paged", "oasr_b200_conformer_chunk_paged_split"])
@pytest.mark.parametrize("change,code", [
    (dict(k_pools=[BASE, None]), _lib.ERR_INVALID), (dict(v_pools=[None, BASE]), _lib.ERR_INVALID), (dict(num_blocks=0), _lib.ERR_INVALID),
    (dict(num_blocks=-3), _lib.ERR_INVALID), (dict(block_size=0), _lib.ERR_INVALID), (dict(blocks_per_seq=0), _lib.ERR_INVALID),
    (dict(pos_proj=BASE + 8), _lib.ERR_ALIGN), (dict(scales=BASE, k_pools=[None, BASE]), _lib.ERR_INVALID)])
def test_a_step_refuses_what_the_page_write_and_the_attention_refuse(entry, change, code):
    """Of few streams as of many, and with both page kinds: a missing pool, an empty page geometry, an unaligned table."""
    a = dict(k_pools=[BASE, BASE], v_pools=[BASE, BASE], num_blocks=8, block_size=16, blocks_per_seq=4, pos_proj=BASE, scales=None)
    a.update(change)
    layers = (_lib.ConformerLayer * 2)()
    model = _lib.ConformerModel(d_model=128, heads=2, ffn=256, kernel=15, num_layers=2, vocab_padded=16, embed_in=256, dtype=_lib.DT_BF16,
                                eps=1e-5, layers=layers, embed_w=BASE, embed_b=BASE, pos_proj=a["pos_proj"], pos_proj_rows=64)
    pools = lambda ps: (ctypes.c_void_p * 2)(*ps)
    with pytest.raises(_lib.OasrB200Error) as e:
        _lib.call(entry, ctypes.byref(model), BASE, 2, 16, pools(a["k_pools"]), pools(a["v_pools"]), BASE, BASE, BASE, BASE,
                  a["blocks_per_seq"], a["block_size"], a["num_blocks"], a["scales"], BASE, 4, BASE, BASE, 1 << 40, BASE, None, None)
    assert e.value.code == code
