"""What the Python binding hands to the library: refusals come back as the library's, and calls that need no array take none.
All of it answers on the host (a stream of handle 0 stands for the current one)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

import b200kv

STREAM = SimpleNamespace(cuda_stream=0)
BF16, I32, U8 = torch.bfloat16, torch.int32, torch.uint8


def _aligned(*shape, dtype=BF16):
    t = torch.zeros(shape, dtype=dtype)
    assert t.data_ptr() % 16 == 0
    return t


def _view():
    return b200kv.pool_view(_aligned(128, 576))


def _append_fused(**k):
    a = dict(view=_view(), kv_a=_aligned(2, 576), gamma=_aligned(512), cos=_aligned(2, 64), sin=_aligned(2, 64), slot_mapping=_aligned(2, dtype=I32))
    b200kv.append_fused(**{**a, **k}, stream=STREAM)


def _gather(**k):
    a = dict(view=_view(), block_table=_aligned(2, 1, dtype=I32), kv_len=_aligned(2, dtype=I32), block_size=64, out_latent=_aligned(4, 512),
             out_rope=_aligned(4, 64), out_row_offsets=_aligned(2, dtype=torch.int64), total_rows=4)
    b200kv.gather(**{**a, **k}, stream=STREAM)


def _indexer(**k):
    a = dict(q_fp8=_aligned(2, 4, 128, dtype=U8), q_scale=_aligned(2, 4, dtype=torch.float32), weights=_aligned(2, 4),
             key_pool=_aligned(128, 128, dtype=U8), k_scale=_aligned(128, dtype=torch.float32), block_table=_aligned(2, 1, dtype=I32),
             kv_len=_aligned(2, dtype=I32), block_size=64, max_kv_len=64, k=8)
    b200kv.indexer_topk(**{**a, **k}, stream=STREAM)


def _decode(call=None, **k):
    a = dict(q=_aligned(2, 64, 576), view=_view(), block_table=_aligned(2, 1, dtype=I32), kv_len=_aligned(2, dtype=I32), block_size=64,
             scale=1.0 / 24.0, out=_aligned(2, 64, 512))
    (call or b200kv.mla_decode)(**{**a, **k}, stream=STREAM)


def _merge(**k):
    a = dict(partial_o=torch.zeros(2, 4, 512), partial_m=torch.zeros(2, 4), partial_l=torch.zeros(2, 4), out=_aligned(4, 512))
    b200kv.lse_merge(**{**a, **k}, stream=STREAM)


@pytest.mark.parametrize("call,name", [(_append_fused, "gamma"), (_gather, "out_row_offsets"), (_indexer, "q_scale"), (_indexer, "weights"),
                                       (_indexer, "k_scale"), (_indexer, "kv_len"), (_decode, "kv_len"), (_decode, "out"),
                                       (_merge, "partial_o"), (_merge, "out")])
def test_a_missing_array_is_the_librarys_refusal(call, name):
    with pytest.raises(b200kv.B200KVError) as refused:
        call(**{name: None})
    assert refused.value.code == b200kv.ERR_NULLPTR


def test_calls_without_work_need_no_arrays():
    none = _aligned(0, dtype=I32)
    b200kv.append(_view(), None, None, none, stream=STREAM)
    _append_fused(kv_a=None, gamma=None, slot_mapping=none)
    _gather(block_table=None, kv_len=none, out_latent=None, out_rope=None, out_row_offsets=none.long(), total_rows=0)


def test_further_dimensions_and_wrong_counts():
    b200kv.lse_merge(torch.zeros(2, 0, 512), torch.zeros(2, 0, 1), torch.zeros(2, 0, 1), _aligned(0, 512), stream=STREAM)
    b200kv.mx_quant_e4m3(_aligned(0, 64, 1), _aligned(0, 64, dtype=U8), _aligned(0, 2, dtype=U8), stream=STREAM)
    t = torch.zeros(2, 64)
    for partial in ((t, t), (t, t, t, t)):
        with pytest.raises(ValueError):
            _decode(partial=partial)
    with pytest.raises(ValueError):
        _decode(new_rows=(_aligned(2, 512), _aligned(2, 64), None))


def test_argument_types_are_checked():
    """The library's functions take a pointer to their own structure (or the structure), and calls a pool view: anything else
    would be read as addresses."""
    wrong = b200kv.KvCache()
    for call in (_append_fused, _decode, lambda **k: _decode(b200kv.mla_decode_static, **k)):
        with pytest.raises(TypeError):
            call(view=wrong)
        with pytest.raises(TypeError):
            call(view=bytes(_view()))
    for name, own, other in (("b200kv_mla_decode", b200kv.DecodeArgs, b200kv.IndexerArgs),
                             ("b200kv_mla_decode_static", b200kv.DecodeArgs, b200kv.ProducerArgs),
                             ("b200kv_append_fused", b200kv.ProducerArgs, b200kv.DecodeArgs),
                             ("b200kv_indexer_topk", b200kv.IndexerArgs, b200kv.ProducerArgs)):
        fn = getattr(b200kv.lib, name)
        for args in (own(), ctypes.byref(own()), None):
            assert fn(args, None, None) != b200kv.ERR_RUNTIME  # taken, and refused or found empty by the library
        for args in (other(), ctypes.byref(other()), bytes(ctypes.sizeof(own)), 4096):
            with pytest.raises(ctypes.ArgumentError):
                fn(args, None, None)
