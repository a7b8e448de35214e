"""The cluster form of the decode attention (one launch, partials exchanged through distributed shared memory): every
cluster size (the batch decides it), every split of a cluster into token ranges and head groups (the length decides it),
tile edges, and the geometries that only this form serves on tensor cores (any block size, any head count)."""
import numpy as np
import pytest
import torch

import b200kv
import kvo
import scenarios
from gpu_util import from_dev_bf16, run_decode, status_ok, to_dev_bf16, to_dev_i32

pytestmark = pytest.mark.gpu

NAN_BF16 = 0x7FC0
EDGES = [1, 63, 64, 65, 128, 129, 192, 257, 320, 513, 640]


def _pool_with_poison(kv_len, bs):
    """A pool whose rows outside the sequences are NaN, and its tables."""
    blocks = int(sum(scenarios.blocks_for(int(n), bs) for n in kv_len)) + 3
    table = scenarios.build_tables(kv_len, bs, blocks, order=kvo.permutation(blocks))
    pool = kvo.make_pool(blocks * bs)
    owned = np.zeros(blocks * bs, dtype=bool)
    for b, n in enumerate(kv_len):
        j = np.arange(int(n))
        owned[table[b, j // bs].astype(np.int64) * bs + j % bs] = True
    owned[0] = True  # (a row past a sequence's end may be read as row 0, whose weight is then zero)
    poisoned = pool.copy()
    poisoned[~owned] = NAN_BF16
    return pool, poisoned, table


# batch -> cluster size: 1 .. 8 sequences 16 (or 8), then 8, 4, 2 and single CTAs
@pytest.mark.parametrize("batch", [1, 2, 7, 12, 30, 60, 140])
def test_small_batches_match_the_reference(batch):
    bs = 64
    kv_len = np.array([([512] + EDGES + [0])[(5 * i + batch) % 13] for i in range(batch)], dtype=np.int32)
    if batch >= 140:
        kv_len = np.minimum(kv_len, 512).astype(np.int32)  # table of eight tiles: still the cluster form with single CTAs
    if not kv_len.any():
        kv_len[0] = 65
    pool, poisoned, table = _pool_with_poison(kv_len, bs)
    q = kvo.make_q(batch, scale=2.0 / 24.0)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, pool, table, kv_len, bs, 1.0 / 24.0)
    out, lse = run_decode(q, poisoned, table, kv_len, bs, 1.0 / 24.0, b200kv.DECODE_TCGEN05)
    scenarios.check_attention(out, lse, ref_out, ref_lse, what=f"cluster batch {batch}")
    assert (out[kv_len == 0] == 0).all()


@pytest.mark.parametrize("length", [1, 64, 100, 129, 257, 512, 513, 1024, 2048, 8192])
def test_one_sequence_of_every_split(length):
    """Up to 2,048 tokens one sequence takes a cluster of 16: 4 x 4, 8 x 2 and 16 x 1 token ranges x head groups (8,192 are the
    other kernel's)."""
    kv_len = np.array([length], dtype=np.int32)
    pool, poisoned, table = _pool_with_poison(kv_len, 128)
    q = kvo.make_q(1)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, pool, table, kv_len, 128, 1.0 / 24.0)
    out, lse = run_decode(q, poisoned, table, kv_len, 128, 1.0 / 24.0, b200kv.DECODE_TCGEN05)
    scenarios.check_attention(out, lse, ref_out, ref_lse, what=f"cluster length {length}", strict_abs=True)
    po, pm, pl = run_decode(q, poisoned, table, kv_len, 128, 1.0 / 24.0, b200kv.DECODE_TCGEN05, partial=True)
    scenarios.check_attention(kvo.f32_to_bf16(po / pl[..., None]), pm + np.log(pl), ref_out, ref_lse,
                              what=f"cluster partial {length}", strict_abs=True)


@pytest.mark.parametrize("kv_len", [[1], [129], [64, 65, 1, 700], [128] * 40])
def test_fused_append_and_quantisation(kv_len):
    """The CTAs of every head group put the new row into their copy of its tile, one of them into the pool; the quantised
    bytes are those of the stand-alone quantiser on the output."""
    bs, batch = 64, len(kv_len)
    kv_len = np.array(kv_len, dtype=np.int32)
    pool, _, table = _pool_with_poison(kv_len, bs)
    latent, rope = kvo.normal_bf16(batch * 512, 21).reshape(batch, 512), kvo.normal_bf16(batch * 64, 22).reshape(batch, 64)
    want = pool.copy()
    last = kv_len.astype(np.int64) - 1
    rows = table[np.arange(batch), last // bs].astype(np.int64) * bs + last % bs
    want[rows, :512], want[rows, 512:] = latent, rope
    q = kvo.make_q(batch)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, want, table, kv_len, bs, 1.0 / 24.0)
    d_pool, status = to_dev_bf16(pool), b200kv.new_status()
    out = torch.empty((batch, 64, 512), dtype=torch.bfloat16, device="cuda")
    lse = torch.empty((batch, 64), dtype=torch.float32, device="cuda")
    fp8 = torch.empty((batch, 64, 512), dtype=torch.uint8, device="cuda")
    scales = torch.empty((batch, 64, 16), dtype=torch.uint8, device="cuda")
    ws = torch.empty(b200kv.decode_workspace_bytes(batch), dtype=torch.uint8, device="cuda")
    b200kv.mla_decode(to_dev_bf16(q), b200kv.pool_view(d_pool), to_dev_i32(table), to_dev_i32(kv_len), bs, 1.0 / 24.0, out=out, lse=lse,
                      workspace=ws, status=status, new_rows=(to_dev_bf16(latent), to_dev_bf16(rope)), stable_tables=True,
                      quantised=(fp8, scales))
    status_ok(status)
    assert np.array_equal(from_dev_bf16(d_pool), want)
    # sequences of one token have outputs of magnitude 3: the per-row bound, not the absolute one
    scenarios.check_attention(from_dev_bf16(out), lse.cpu().numpy(), ref_out, ref_lse, what="cluster append")
    fp8_2, scales_2 = torch.empty((batch, 64 * 512), dtype=torch.uint8, device="cuda"), torch.empty((batch, 1024), dtype=torch.uint8, device="cuda")
    b200kv.mx_quant_e4m3(out.view(batch, -1), fp8_2, scales_2)
    assert torch.equal(fp8.view(batch, -1), fp8_2) and torch.equal(scales.view(batch, -1), scales_2)


@pytest.mark.parametrize("heads,bs", [(64, 16), (64, 1), (64, 48), (64, 96), (1, 64), (5, 16), (16, 64), (63, 32), (65, 64), (128, 16)])
def test_any_geometry_is_as_exact_as_the_cuda_core_kernel(heads, bs):
    """Block sizes that are no multiple of 64 and head counts other than 64: against the float64 reference, and no
    further from it than the CUDA-core kernel with its fp32 weights. Both results are bf16, whose rounding is 2^-9 of a
    value at most; the split weights add 2^-17, so the mean errors agree far within 10 %."""
    kv_len = np.array([1, 17, 64, 65, 1000, 0, 333], dtype=np.int32)
    pool, poisoned, table = _pool_with_poison(kv_len, bs)
    q = kvo.make_q(len(kv_len), heads=heads, scale=0.3)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, pool, table, kv_len, bs, 1.0 / 24.0)
    out, lse = run_decode(q, poisoned, table, kv_len, bs, 1.0 / 24.0, b200kv.DECODE_AUTO)
    scenarios.check_attention(out, lse, ref_out, ref_lse, what=f"any geometry {heads} x {bs}")
    simt, _ = run_decode(q, poisoned, table, kv_len, bs, 1.0 / 24.0, b200kv.DECODE_SIMT)
    live = kv_len > 0
    err = np.abs(kvo.bf16_to_f32(out[live]).astype(np.float64) - ref_out[live]).mean()
    err_simt = np.abs(kvo.bf16_to_f32(simt[live]).astype(np.float64) - ref_out[live]).mean()
    assert err <= 1.1 * err_simt, (err, err_simt)


def test_any_geometry_reports_a_length_beyond_the_table():
    bs = 16
    pool, _, table = _pool_with_poison(np.array([200, 64], dtype=np.int32), bs)
    status = b200kv.new_status()
    out = torch.empty((2, 64, 512), dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(b200kv.decode_workspace_bytes(2), dtype=torch.uint8, device="cuda")
    b200kv.mla_decode(to_dev_bf16(kvo.make_q(2)), b200kv.pool_view(to_dev_bf16(pool)), to_dev_i32(table),
                      to_dev_i32([200, bs * table.shape[1] + 40]), bs, 1.0 / 24.0, out=out, workspace=ws, status=status)
    torch.cuda.synchronize()
    got = status.cpu().tolist()
    assert got[0] == b200kv.DEV_BAD_BLOCK and got[1] == 1, got


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 6, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("quantised", [False, True])
def test_merge_of_many_parts_in_every_shape(batch, quantised):
    """Histories beyond the cluster form's: partials of every CTA, merged in the shape that the batch selects. Against the
    CUDA-core kernel (fp32 weights, its own merge): bf16 results of the same rows, whose weights the tensor-core kernel
    rounds to bf16 (2^-9 of values of magnitude 4 at most)."""
    bs = 64
    kv_len = np.array([9000 - 517 * (i % 9) if i != 1 else 65 for i in range(batch)], dtype=np.int32)
    blocks = int(sum(scenarios.blocks_for(int(n), bs) for n in kv_len)) + 3
    table = scenarios.build_tables(kv_len, bs, blocks, order=kvo.permutation(blocks))
    g = torch.Generator(device="cuda")
    g.manual_seed(batch)
    pool = torch.randn((blocks * bs, 576), generator=g, device="cuda").bfloat16()
    q = torch.randn((batch, 64, 576), generator=g, device="cuda").bfloat16()
    d_table, d_len = to_dev_i32(table), to_dev_i32(kv_len)
    ws = torch.empty(b200kv.decode_workspace_bytes(batch), dtype=torch.uint8, device="cuda")
    status = b200kv.new_status()
    got = []
    for variant in (b200kv.DECODE_TCGEN05, b200kv.DECODE_SIMT):
        out = torch.full((batch, 64, 512), float("nan"), dtype=torch.bfloat16, device="cuda")
        lse = torch.full((batch, 64), float("nan"), dtype=torch.float32, device="cuda")
        codes = (torch.zeros((batch, 64, 512), dtype=torch.uint8, device="cuda"), torch.zeros((batch, 64, 16), dtype=torch.uint8, device="cuda"))
        b200kv.mla_decode(q, b200kv.pool_view(pool), d_table, d_len, bs, 1.0 / 24.0, out=out, lse=lse, workspace=ws, status=status,
                          variant=variant, quantised=codes if quantised else None)
        status_ok(status)
        got.append((out.float(), lse))
        if quantised:
            fp8, scales = torch.empty((batch, 64 * 512), dtype=torch.uint8, device="cuda"), torch.empty((batch, 1024), dtype=torch.uint8, device="cuda")
            b200kv.mx_quant_e4m3(out.view(batch, -1), fp8, scales)
            assert torch.equal(codes[0].view(batch, -1), fp8) and torch.equal(codes[1].view(batch, -1), scales)
    assert ((got[0][0] - got[1][0]).abs() <= 2e-3 + 1e-2 * got[1][0].abs().amax(dim=2, keepdim=True)).all()
    assert ((got[0][1] - got[1][1]).abs() <= 1e-4).all()


def _decode_dev(q, pool, table, kv_len, bs, variant=b200kv.DECODE_AUTO, partial=False, max_ctas=0):
    """The call on torch tensors: (out, lse), or (o, m, l) of a partial."""
    batch, heads = q.shape[:2]
    ws = torch.empty(b200kv.decode_workspace_bytes(batch, heads, max_ctas), dtype=torch.uint8, device="cuda")
    status = b200kv.new_status()
    if partial:
        got = (torch.zeros((batch, heads, 512), device="cuda"), torch.zeros((batch, heads), device="cuda"), torch.zeros((batch, heads), device="cuda"))
        kw = {"partial": got}
    else:
        got = (torch.zeros((batch, heads, 512), dtype=torch.bfloat16, device="cuda"), torch.zeros((batch, heads), device="cuda"))
        kw = {"out": got[0], "lse": got[1]}
    b200kv.mla_decode(q, b200kv.pool_view(pool), table, kv_len, bs, 1.0 / 24.0, workspace=ws, status=status, variant=variant,
                      max_ctas=max_ctas, **kw)
    status_ok(status)
    return got


def _case(kv_len, bs, heads=64, seed=3):
    kv_len = np.array(kv_len, dtype=np.int32)
    blocks = int(sum(scenarios.blocks_for(int(n), bs) for n in kv_len)) + 3
    table = scenarios.build_tables(kv_len, bs, blocks, order=kvo.permutation(blocks))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    pool = torch.randn((blocks * bs, 576), generator=g, device="cuda").bfloat16()
    q = torch.randn((len(kv_len), heads, 576), generator=g, device="cuda").bfloat16()
    rows = [torch.from_numpy(table[b, np.arange(n) // bs].astype(np.int64) * bs + np.arange(n) % bs).cuda() for b, n in enumerate(kv_len)]
    return q, pool, to_dev_i32(table), to_dev_i32(kv_len), rows


def _attention_f64(q, pool, rows):
    out, lse = [], []
    for b, r in enumerate(rows):
        kv = pool[r].double()
        s = q[b].double() @ kv.T / 24.0
        lse.append(torch.logsumexp(s, dim=1))
        out.append(torch.softmax(s, dim=1) @ kv[:, :512])
    return torch.stack(out), torch.stack(lse)


# (lengths, block size, heads): clusters of 16, of one and several head groups, of 8 and of 4, single CTAs, other geometries
NOT_FINITE = [([700], 64, 64), ([2048], 64, 64), ([100, 64, 513], 64, 64), ([300] * 20, 64, 64), ([500] * 140, 64, 64),
              ([700, 65], 16, 64), ([333], 1, 16), ([400] * 150, 64, 16),
              # the flat kernel: sequences cut over many CTAs and merged in several shapes, and whole ones beside a long one
              ([9000], 64, 64), ([9000, 5000, 300], 64, 64), ([3000] * 12, 64, 64), ([9000] + [100] * 200, 64, 64)]


@pytest.mark.parametrize("kv_len,bs,heads", NOT_FINITE)
@pytest.mark.parametrize("at", ["first", "last"])
def test_a_nan_in_a_sequence_makes_its_rows_nan(kv_len, bs, heads, at):
    """However many CTAs share the sequence out; the other sequences are what they were. (The NaN sits in the rotary part of
    one token's key, so it reaches a row through that token's weight only.)"""
    q, pool, table, lens, rows = _case(kv_len, bs, heads)
    clean, clean_lse = _decode_dev(q, pool, table, lens, bs)
    hit = len(kv_len) // 2
    pool[rows[hit][0 if at == "first" else -1], 575] = float("nan")
    out, lse = _decode_dev(q, pool, table, lens, bs)
    assert out[hit].isnan().all() and lse[hit].isnan().all()
    rest = torch.arange(len(kv_len), device="cuda") != hit
    assert torch.equal(out[rest], clean[rest]) and torch.equal(lse[rest], clean_lse[rest])
    if heads == 64 and bs % 64 == 0:
        _, _, l = _decode_dev(q, pool, table, lens, bs, partial=True)
        assert l[hit].isnan().all() and l[rest].isfinite().all()


@pytest.mark.parametrize("kv_len,bs,heads", NOT_FINITE)
def test_scores_of_minus_infinity_have_no_weight(kv_len, bs, heads):
    """Tokens whose scores are all -infinity at the beginning of a sequence, past the first tile, count for nothing; a
    sequence of nothing else is empty. (An infinity in the rotary part of the keys against a negative query.)"""
    q, pool, table, lens, rows = _case(kv_len, bs, heads)
    q[:, :, 575] = -1.0
    dead = [min(len(r) - 1, 130) for r in rows]
    for r, n in zip(rows, dead):
        pool[r[:n], 575] = float("inf")
    want, want_lse = _attention_f64(q, pool, [r[n:] for r, n in zip(rows, dead)])
    out, lse = _decode_dev(q, pool, table, lens, bs)
    assert ((out.double() - want).abs() <= 2e-3 + 1e-2 * want.abs().amax(dim=2, keepdim=True)).all()
    assert (lse.double() - want_lse).abs().max() <= 1e-4
    hit = len(kv_len) // 2
    pool[rows[hit], 575] = float("inf")
    out, lse = _decode_dev(q, pool, table, lens, bs)
    assert (out[hit] == 0).all() and (lse[hit] == float("-inf")).all()


@pytest.mark.parametrize("gain", [1.0, 3.0])
def test_log_sum_exp_of_any_geometry_is_as_exact_as_the_cuda_core_kernels(gain):
    """Against float64, over lengths, head counts and block sizes together: the root mean square of the tensor cores' sums
    and of the fp32 chains differ by the luck of their roundings (both are close to that of the fp32 result itself), so by
    less than a tenth."""
    squares = {b200kv.DECODE_AUTO: [], b200kv.DECODE_SIMT: []}
    for seed in range(3):
        for kv_len in ([1, 17, 64, 65, 1000, 333], [4096, 3000], [8192]):
            for heads, bs in ((64, 16), (64, 1), (16, 64), (128, 8)):
                q, pool, table, lens, rows = _case(kv_len, bs, heads, seed)
                q = (q.float() * gain).bfloat16()
                _, want = _attention_f64(q, pool, rows)
                for variant, errors in squares.items():
                    _, lse = _decode_dev(q, pool, table, lens, bs, variant)
                    errors.append((lse.double() - want).pow(2).mean(1))
    auto, simt = (torch.cat(squares[v]).mean().sqrt().item() for v in (b200kv.DECODE_AUTO, b200kv.DECODE_SIMT))
    assert auto <= 1.1 * simt, (auto, simt)


@pytest.mark.parametrize("batch,longest", [(40, 750), (140, 512)])
def test_fused_append_where_a_cta_has_several_tiles(batch, longest):
    """The new row goes into a stage that has been filled before; bf16 output alone (quantised calls come here with a tile a
    CTA only). Rows at the beginning, in the middle and at the end of tiles; the pool bit for bit."""
    bs = 64
    kv_len = np.array([[longest, longest // 64 * 64, longest // 64 * 64 - 63, 300, 449, 129, 1, 64, 65, 257][i % 10] for i in range(batch)], dtype=np.int32)
    pool, poisoned, table = _pool_with_poison(kv_len, bs)
    latent, rope = kvo.normal_bf16(batch * 512, 21).reshape(batch, 512), kvo.normal_bf16(batch * 64, 22).reshape(batch, 64)
    last = kv_len.astype(np.int64) - 1
    rows = table[np.arange(batch), last // bs].astype(np.int64) * bs + last % bs
    whole, want = pool.copy(), poisoned.copy()
    for p in (whole, want):
        p[rows, :512], p[rows, 512:] = latent, rope
    q = kvo.make_q(batch)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, whole, table, kv_len, bs, 1.0 / 24.0)
    for max_ctas in (0, 5):  # and the kernel for many tiles
        d_pool, status = to_dev_bf16(poisoned), b200kv.new_status()
        out = torch.empty((batch, 64, 512), dtype=torch.bfloat16, device="cuda")
        lse = torch.empty((batch, 64), dtype=torch.float32, device="cuda")
        ws = torch.empty(b200kv.decode_workspace_bytes(batch, 64, max_ctas), dtype=torch.uint8, device="cuda")
        b200kv.mla_decode(to_dev_bf16(q), b200kv.pool_view(d_pool), to_dev_i32(table), to_dev_i32(kv_len), bs, 1.0 / 24.0, out=out, lse=lse,
                          workspace=ws, status=status, new_rows=(to_dev_bf16(latent), to_dev_bf16(rope)), max_ctas=max_ctas)
        status_ok(status)
        assert np.array_equal(from_dev_bf16(d_pool), want)
        scenarios.check_attention(from_dev_bf16(out), lse.cpu().numpy(), ref_out, ref_lse, what=f"append, several tiles, max_ctas {max_ctas}")


@pytest.mark.parametrize("heads,bs", [(64, 16), (64, 48), (16, 64), (16, 16), (65, 1)])
@pytest.mark.parametrize("two_arrays", [False, True])
def test_shards_and_strided_queries_of_any_geometry(heads, bs, two_arrays):
    """Shards that begin anywhere (out and lse of a range that starts past the first tokens), queries that are slices of wider
    rows with the heads outermost, and latent and rope in arrays of their own."""
    begin = np.array([0, 48, 100, 1, 333], dtype=np.int32)
    length = np.array([64, 200, 1, 0, 700], dtype=np.int32)
    pool, _, table = _pool_with_poison(begin + np.maximum(length, 1), bs)
    q = kvo.make_q(len(length), heads=heads, scale=0.3)
    ref_out, ref_lse = scenarios.ref_attention_f64(q, pool, table, length, bs, 1.0 / 24.0, kv_begin=begin)
    d_pool = to_dev_bf16(pool)
    wide = torch.full((len(pool), 640), float("nan"), dtype=torch.bfloat16, device="cuda")
    wide[:, :512] = d_pool[:, :512]
    rope = d_pool[:, 512:].contiguous()
    view = b200kv.pool_view(wide[:, :512], rope) if two_arrays else b200kv.pool_view(d_pool)
    by_head = torch.full((heads, len(length), 640), float("nan"), dtype=torch.bfloat16, device="cuda")
    by_head[:, :, 64:] = to_dev_bf16(q).transpose(0, 1)
    d_q = by_head.transpose(0, 1)[:, :, 64:]
    out = torch.full((len(length), heads, 512), float("nan"), dtype=torch.bfloat16, device="cuda")
    lse = torch.full((len(length), heads), float("nan"), dtype=torch.float32, device="cuda")
    status = b200kv.new_status()
    ws = torch.empty(b200kv.decode_workspace_bytes(len(length), heads), dtype=torch.uint8, device="cuda")
    b200kv.mla_decode(d_q, view, to_dev_i32(table), to_dev_i32(length), bs, 1.0 / 24.0, out=out, lse=lse, kv_begin=to_dev_i32(begin),
                      workspace=ws, status=status)
    status_ok(status)
    scenarios.check_attention(from_dev_bf16(out), lse.cpu().numpy(), ref_out, ref_lse, what=f"shards {heads} x {bs}")


@pytest.mark.parametrize("bs", [16, 48, 1])
def test_quantised_output_of_any_block_size(bs):
    """The quantised bytes are those of the stand-alone quantiser on the output, and of the CUDA-core path's wherever the two
    kernels' bf16 agree on a block of 32."""
    kv_len = np.array([1, 70, 1000, 0, 333], dtype=np.int32)
    pool, _, table = _pool_with_poison(kv_len, bs)
    q, batch = to_dev_bf16(kvo.make_q(len(kv_len))), len(kv_len)
    ws = torch.empty(b200kv.decode_workspace_bytes(batch), dtype=torch.uint8, device="cuda")
    got = []
    for variant in (b200kv.DECODE_AUTO, b200kv.DECODE_SIMT):
        out = torch.empty((batch, 64, 512), dtype=torch.bfloat16, device="cuda")
        fp8 = torch.empty((batch, 64, 512), dtype=torch.uint8, device="cuda")
        scales = torch.empty((batch, 64, 16), dtype=torch.uint8, device="cuda")
        status = b200kv.new_status()
        b200kv.mla_decode(q, b200kv.pool_view(to_dev_bf16(pool)), to_dev_i32(table), to_dev_i32(kv_len), bs, 1.0 / 24.0, out=out, workspace=ws,
                          status=status, variant=variant, quantised=(fp8, scales))
        status_ok(status)
        fp8_2, scales_2 = torch.empty((batch, 64 * 512), dtype=torch.uint8, device="cuda"), torch.empty((batch, 1024), dtype=torch.uint8, device="cuda")
        b200kv.mx_quant_e4m3(out.view(batch, -1), fp8_2, scales_2)
        assert torch.equal(fp8.view(batch, -1), fp8_2) and torch.equal(scales.view(batch, -1), scales_2)
        got.append((out.view(-1, 32), fp8.view(-1, 32)))
    same = (got[0][0] == got[1][0]).all(1)
    assert same.float().mean() > 0.8 and torch.equal(got[0][1][same], got[1][1][same])


def test_two_sequences_of_up_to_4096_tokens():
    """The longest sequences that clusters of sixteen take (two of 64 tiles), and one tile more, which they do not."""
    for longest in (2049, 3000, 4096, 4160):
        kv_len = [longest, longest - 777]
        q, pool, table, lens, rows = _case(kv_len, 64)
        want, want_lse = _attention_f64(q, pool, rows)
        out, lse = _decode_dev(q, pool, table, lens, 64)
        assert ((out.double() - want).abs() <= 2e-3 + 1e-2 * want.abs().amax(dim=2, keepdim=True)).all()
        assert (lse.double() - want_lse).abs().max() <= 1e-4


@pytest.mark.parametrize("batch,tiles", [(1, 32), (2, 64), (5, 32), (12, 16), (30, 16), (60, 12), (140, 8)])
def test_which_kernel_takes_a_call(batch, tiles):
    """Up to so many tiles in the longest sequence a table can hold, a call runs in clusters, which leave the workspace alone;
    with one more it runs in the kernel for many tiles, whose sequences are cut and leave partials there."""
    for more in (0, 1):
        q, pool, table, lens, rows = _case([64 * (tiles + more)] * batch, 64)
        ws = torch.full((b200kv.decode_workspace_bytes(batch),), 0x5A, dtype=torch.uint8, device="cuda")
        status = b200kv.new_status()
        out = torch.empty((batch, 64, 512), dtype=torch.bfloat16, device="cuda")
        b200kv.mla_decode(q, b200kv.pool_view(pool), table, lens, 64, 1.0 / 24.0, out=out, workspace=ws, status=status)
        status_ok(status)
        assert bool((ws == 0x5A).all()) == (more == 0)
