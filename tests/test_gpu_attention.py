"""Causal attention against the f16 KV cache, SelfAttention and the whole Block on the GPU, against the oracle's
restatement of the portable arm (src/kernels/kv_attention.rs:155-331) and against their own parts (restating
tests/correctness/model.rs:80-206 in spirit: prefill then decode agree, the block equals its halves)."""
import numpy as np
import pytest
import torch

import oracle as orc
import sme_gemm_b200 as sg
from gpu_util import bits_of, max_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_f32", [True, False])
@pytest.mark.parametrize("heads,kv_heads,hd,start,rows", [(4, 4, 64, 0, 1), (8, 2, 32, 5, 3), (6, 3, 128, 17, 40), (2, 1, 256, 100, 1),
                                                         (3, 1, 8, 0, 9), (32, 8, 128, 300, 2)])
def test_attention_matches_the_scalar_statement(heads, kv_heads, hd, start, rows, q_f32):
    rng = np.random.default_rng(heads * 1000 + start + rows)
    cache = sg.KvCache(heads, kv_heads, hd, start + rows + 3)
    k16 = (rng.standard_normal((start + rows, kv_heads * hd)) * 0.7).astype(np.float16)
    v16 = rng.standard_normal((start + rows, kv_heads * hd)).astype(np.float16)
    cache.extend(torch.from_numpy(k16).cuda(), torch.from_numpy(v16).cuda())
    assert cache.len() == start + rows and not cache.is_empty() and cache.row_len() == kv_heads * hd
    q32 = rng.standard_normal((rows, heads * hd)).astype(np.float32)
    if not q_f32:
        q32 = q32.astype(np.float16).astype(np.float32)
    q = torch.from_numpy(q32 if q_f32 else q32.astype(np.float16)).cuda()
    out = torch.zeros((rows, heads * hd), dtype=torch.float32, device="cuda")
    if rows == 1:
        cache.attend(q, out)
    else:
        cache.attend_causal(q, rows, out)
    want = orc.attention_kv_causal(q32, k16.view(np.uint16), v16.view(np.uint16), start, rows, heads, kv_heads, hd, cache.scale())
    # same products and sums in the same order; the device's expf and the order of the probabilities' sum differ
    assert max_rel(out.cpu().numpy(), want) <= 2e-5
    assert sg.last_status() == 0


def test_cache_bookkeeping_and_refusals():
    cache = sg.KvCache(4, 2, 16, 5).with_scale(0.5)
    assert cache.scale() == 0.5 and cache.capacity() == 5 and cache.query_len() == 64 and cache.is_empty()
    row = torch.ones((2, 32), dtype=torch.float16, device="cuda")
    cache.push(row, row)
    cache.extend(row, row)
    assert cache.len() == 4 and tuple(cache.keys().shape) == (4, 32)
    with pytest.raises(AssertionError, match="KvCache full: 4 \\+ 2 rows over capacity 5"):
        cache.extend(row, row)
    cache.truncate(1)
    assert cache.len() == 1
    out = torch.zeros(64, dtype=torch.float32, device="cuda")
    with pytest.raises(AssertionError, match="attend_causal: 3 rows but 1 cached"):
        cache.attend_causal(torch.zeros((3, 64), device="cuda"), 3, torch.zeros((3, 64), device="cuda"))
    cache.clear()
    with pytest.raises(AssertionError, match="needs at least one cached key"):
        cache.attend(torch.zeros(64, device="cuda"), out)
    with pytest.raises(AssertionError, match="head_dim must be a multiple of 8"):
        sg.KvCache(2, 2, 12, 4)
    with pytest.raises(AssertionError, match="positive multiple of kv_heads"):
        sg.KvCache(5, 2, 16, 4)
    L = sg.lib()
    z = torch.zeros(64, device="cuda")
    k = torch.zeros((4, 32), dtype=torch.float16, device="cuda")
    assert L.smeg_attn_kv_causal_dev(out.data_ptr(), z.data_ptr(), 1, 64, k.data_ptr(), k.data_ptr(), 0, 1, 4, 2, 12, 0.5, 0) == -4
    assert L.smeg_attn_kv_causal_dev(out.data_ptr(), z.data_ptr(), 1, 64, k.data_ptr(), k.data_ptr(), 0, 1, 5, 2, 16, 0.5, 0) == -4


def _attention_parts(rng, d, heads, kv_heads, hd):
    w_qkv = (rng.standard_normal(((heads + 2 * kv_heads) * hd, d)) * 0.08).astype(np.float32)
    w_out = (rng.standard_normal((d, heads * hd)) * 0.08).astype(np.float32)
    qkv = sg.Linear.quantize(w_qkv, sg.WeightLayout.OutIn, w_qkv.shape[0], d)
    out = sg.Linear.quantize(w_out, sg.WeightLayout.OutIn, d, heads * hd)
    return sg.SelfAttention.new(qkv, out, heads, kv_heads, hd), w_qkv, w_out


@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 4, 32), (8, 2, 16)])
def test_self_attention_against_the_oracle_chain_and_prefill_then_decode(heads, kv_heads, hd):
    rng = np.random.default_rng(heads + hd)
    d = 128
    attn, w_qkv, w_out = _attention_parts(rng, d, heads, kv_heads, hd)
    m = 21
    x16 = rng.standard_normal((m + 1, d)).astype(np.float16)
    y0 = rng.standard_normal((m + 1, d)).astype(np.float32)
    # prefill m rows, then one more row against the same cache
    cache = attn.cache(64)
    y = torch.from_numpy(y0.copy()).cuda()
    attn.accumulate(torch.from_numpy(x16[:m]).cuda(), cache, y[:m], m)
    attn.accumulate(torch.from_numpy(x16[m:]).cuda(), cache, y[m:], 1)
    assert cache.len() == m + 1
    # all m + 1 rows at once
    cache2 = attn.cache(64)
    y2 = torch.from_numpy(y0.copy()).cuda()
    attn.accumulate(torch.from_numpy(x16).cuda(), cache2, y2, m + 1)
    # (the one-row projection runs on the decode kernel, the block on the GEMM: the cached rows agree to an f16 rounding)
    assert max_rel(cache.keys().float().cpu().numpy(), cache2.keys().float().cpu().numpy()) <= 2e-3
    assert max_rel(cache.values().float().cpu().numpy(), cache2.values().float().cpu().numpy()) <= 2e-3
    assert max_rel(y.cpu().numpy(), y2.cpu().numpy()) <= 2e-3        # decode GEMV and prefill GEMM kernels differ in summation order
    # the oracle's chain: Q4 projection, scalar attention, Q4 projection, residual add
    q_len, kv_len = heads * hd, kv_heads * hd
    qq, qs, _ = orc.q4_quantize(w_qkv, 0, w_qkv.shape[0], d)
    oq, os_, _ = orc.q4_quantize(w_out, 0, d, q_len)
    xb = x16.view(np.uint16)
    qkv_o = orc.f16_bits_to_f32(orc.matmul_q4(xb, qq, qs, None, w_qkv.shape[0], d, 32, m + 1)).reshape(m + 1, -1)
    kb = orc.f32_to_f16_bits(qkv_o[:, q_len:q_len + kv_len])
    vb = orc.f32_to_f16_bits(qkv_o[:, q_len + kv_len:])
    att = orc.attention_kv_causal(qkv_o[:, :q_len], kb, vb, 0, m + 1, heads, kv_heads, hd, cache.scale())
    out_o = orc.f16_bits_to_f32(orc.matmul_q4(orc.f32_to_f16_bits(att), oq, os_, None, d, q_len, 32, m + 1)).reshape(m + 1, d)
    assert max_rel(y2.cpu().numpy(), y0 + out_o) <= 1e-2
    assert sg.last_status() == 0


@pytest.mark.parametrize("rows", [1, 5, 70])
def test_block_equals_its_halves(rows):
    """Block::accumulate (src/block.rs:90-106): norm1 -> attention -> norm2 -> MLP, the same bits as the parts run in turn."""
    rng = np.random.default_rng(rows)
    d, heads, hd, f = 128, 4, 32, 384
    attn, _, _ = _attention_parts(rng, d, heads, heads, hd)
    up = sg.Linear.quantize((rng.standard_normal((f, d)) * 0.05).astype(np.float32), sg.WeightLayout.OutIn, f, d)
    down = sg.Linear.quantize((rng.standard_normal((d, f)) * 0.05).astype(np.float32), sg.WeightLayout.OutIn, d, f)
    n1 = sg.Norm.layer(rng.uniform(0.5, 1.5, d).astype(np.float32), (rng.standard_normal(d) * 0.1).astype(np.float32), 1e-5)
    n2 = sg.Norm.rms(rng.uniform(0.5, 1.5, d).astype(np.float32), 1e-5)
    block = sg.Block.new(n1, attn, n2, sg.Mlp.new(up, sg.Gate.Gelu, down))
    x0 = rng.standard_normal((rows, d)).astype(np.float32)
    cache = block.cache(128)
    warm = torch.from_numpy(rng.standard_normal((3, d)).astype(np.float32)).cuda()
    block.accumulate(warm, cache, 3)                               # three earlier positions
    x = torch.from_numpy(x0.copy()).cuda()
    block.accumulate(x, cache, rows)
    assert cache.len() == 3 + rows
    # the parts, on a cache with the same three positions
    cache2 = block.cache(128)
    cache2.extend(cache.keys()[:3].clone(), cache.values()[:3].clone())
    xp = torch.from_numpy(x0.copy()).cuda()
    h = torch.empty((rows, d), dtype=torch.float16, device="cuda")
    n1.forward(xp, h)
    attn.accumulate(h, cache2, xp, rows)
    n2.forward(xp, h)
    block.mlp.accumulate(h, xp, rows)
    assert torch.equal(x, xp)
    assert torch.isfinite(x).all() and sg.last_status() == 0


def test_two_layer_model_from_a_checkpoint_file(tmp_path):
    """A safetensors file -> Checkpoint -> Blocks (examples/shakespeare/model.rs:84-125 in small): a prompt through both
    layers against the oracle's chain on the same quantised weights, then decode steps against re-running the longer prompt."""
    from sme_gemm_b200.checkpoint import Checkpoint
    from test_checkpoint import write_safetensors
    rng = np.random.default_rng(42)
    d, heads, hd, ff, layers = 64, 2, 32, 256, 2
    tensors = {}
    for i in range(layers):
        p = f"transformer.h.{i}."
        tensors[p + "ln_1.weight"] = ("F32", rng.uniform(0.5, 1.5, d).astype("<f4"))
        tensors[p + "ln_2.weight"] = ("F32", rng.uniform(0.5, 1.5, d).astype("<f4"))
        tensors[p + "attn.c_attn.weight"] = ("F32", (rng.standard_normal((3 * d, d)) * 0.1).astype("<f4"))
        tensors[p + "attn.c_proj.weight"] = ("F32", (rng.standard_normal((d, d)) * 0.1).astype("<f4"))
        tensors[p + "mlp.c_fc.weight"] = ("F32", (rng.standard_normal((ff, d)) * 0.1).astype("<f4"))
        tensors[p + "mlp.c_proj.weight"] = ("F32", (rng.standard_normal((d, ff)) * 0.1).astype("<f4"))
    path = tmp_path / "model.safetensors"
    path.write_bytes(write_safetensors(tensors, {"format": "pt"}))
    ck = Checkpoint.load(path)
    blocks = []
    for i in range(layers):
        p = f"transformer.h.{i}."
        blocks.append(sg.Block.new(ck.norm(p + "ln_1.weight"),
                                   sg.SelfAttention.new(ck.linear(p + "attn.c_attn.weight"), ck.linear(p + "attn.c_proj.weight"), heads, heads, hd),
                                   ck.norm(p + "ln_2.weight"),
                                   sg.Mlp.new(ck.linear(p + "mlp.c_fc.weight"), sg.Gate.Gelu, ck.linear(p + "mlp.c_proj.weight"))))
    rows, extra = 20, 3
    x0 = rng.standard_normal((rows + extra, d)).astype(np.float32)

    def run(n_prefill, n_decode):
        caches = [b.cache(64) for b in blocks]
        x = torch.from_numpy(x0[:n_prefill].copy()).cuda()
        for b, c in zip(blocks, caches):
            b.accumulate(x, c, n_prefill)
        outs = [x]
        for s in range(n_decode):
            xs = torch.from_numpy(x0[n_prefill + s:n_prefill + s + 1].copy()).cuda()
            for b, c in zip(blocks, caches):
                b.accumulate(xs, c, 1)
            outs.append(xs)
        return torch.cat(outs).cpu().numpy()

    got = run(rows, extra)
    whole = run(rows + extra, 0)
    assert max_rel(got, whole) <= 5e-3                                # prefill + decode steps == the longer prompt
    # the oracle's chain for the prompt
    x = x0[:rows].copy()
    scale = float(np.float32(1.0) / np.sqrt(np.float32(hd)))
    for i in range(layers):
        p = f"transformer.h.{i}."
        def lin(name, a_bits, m, nodes=None):
            w, n, k = ck.matrix(p + name)
            q, s, _ = orc.q4_quantize(w, 0, n, k)
            return orc.matmul_q4(a_bits, q, s, None, n, k, 32, m, nodes)
        h16, _ = orc.norm_rows(x, ck.get(p + "ln_1.weight"), None, 1e-5, False)
        qkv = orc.f16_bits_to_f32(lin("attn.c_attn.weight", h16, rows)).reshape(rows, 3 * d)
        att = orc.attention_kv_causal(qkv[:, :d], orc.f32_to_f16_bits(qkv[:, d:2 * d]), orc.f32_to_f16_bits(qkv[:, 2 * d:]), 0, rows,
                                      heads, heads, hd, scale)
        x = x + orc.f16_bits_to_f32(lin("attn.c_proj.weight", orc.f32_to_f16_bits(att), rows)).reshape(rows, d)
        h16, _ = orc.norm_rows(x, ck.get(p + "ln_2.weight"), None, 1e-5, False)
        hid = lin("mlp.c_fc.weight", h16, rows, orc.Nodes([(8, int(sg.Gate.Gelu), 0.0, None, 0)]))
        x = x + orc.f16_bits_to_f32(lin("mlp.c_proj.weight", hid, rows)).reshape(rows, d)
    assert max_rel(got[:rows], x) <= 2e-2
    assert sg.last_status() == 0


@pytest.mark.parametrize("m", [1, 3, 5, 70])
def test_partial_product_is_the_projection_before_its_rounding(m):
    """Linear.partial (one rank's share of a projection split over its input width): the f32 sums whose f16 rounding is
    the projection's output; and a one-rank TpSelfAttention is the block itself."""
    from sme_gemm_b200.tp import TpSelfAttention
    rng = np.random.default_rng(31)
    d, heads, kv_heads, hd = 256, 8, 4, 32
    wo = (rng.standard_normal((d, heads * hd)) * 0.05).astype(np.float32)
    wq = (rng.standard_normal(((heads + 2 * kv_heads) * hd, d)) * 0.05).astype(np.float32)
    out = sg.Linear.quantize(wo, sg.WeightLayout.OutIn, d, heads * hd)
    a = torch.from_numpy(rng.standard_normal((m, heads * hd)).astype(np.float16)).cuda()
    part = torch.zeros((m, d), dtype=torch.float32, device="cuda")
    c = torch.zeros((m, d), dtype=torch.float16, device="cuda")
    out.partial(a, part, m)
    out.forward(a, c, m)
    torch.cuda.synchronize()
    assert max_rel(part.cpu().numpy(), c.float().cpu().numpy()) <= 1e-3
    deq = orc.f16_bits_to_f32(orc.q4_dequant(*orc.q4_quantize(wo, 0, d, heads * hd)[:2], None, d, heads * hd)).reshape(heads * hd, d)
    ref = a.cpu().numpy().astype(np.float64) @ deq.astype(np.float64)
    assert max_rel(part.cpu().numpy(), ref.astype(np.float32)) <= 2e-3
    with pytest.raises(AssertionError, match="plain Q4 weights"):
        sg.Linear.quantize(wo, sg.WeightLayout.OutIn, d, heads * hd, bias=np.zeros(d, np.float16)).partial(a, part, m)
    # world = 1: the tensor-parallel block is the block
    tp = TpSelfAttention.quantize(wq, wo, heads, kv_heads, hd, 0, 1)
    one = sg.SelfAttention(sg.Linear.quantize(wq, sg.WeightLayout.OutIn, wq.shape[0], d), out, heads, kv_heads, hd)
    x = torch.from_numpy(rng.standard_normal((m, d)).astype(np.float16)).cuda()
    y0 = torch.from_numpy(rng.standard_normal((m, d)).astype(np.float32)).cuda()
    y1, y2 = y0.clone(), y0.clone()
    tp.accumulate(x, tp.cache(128), y1, m)
    one.accumulate(x, one.cache(128), y2, m)
    torch.cuda.synchronize()
    assert torch.equal(y1, y2) and sg.last_status() == 0


@pytest.mark.parametrize("heads,kv_heads,hd,start,rows,q_f32,pad", [
    (4, 2, 64, 127, 1, False, 0), (4, 2, 64, 128, 1, True, 0), (8, 2, 128, 1023, 1, False, 16), (8, 1, 128, 4095, 1, False, 0),
    (6, 2, 72, 300, 5, False, 8), (4, 4, 256, 600, 3, True, 0), (6, 2, 200, 130, 70, False, 3), (1, 1, 64, 0, 129, False, 0),
    (12, 4, 64, 250, 200, False, 64), (5, 1, 48, 511, 77, True, 0), (32, 8, 128, 0, 512, False, 2048), (32, 8, 128, 385, 130, False, 0)])
def test_attention_tiles_splits_and_ragged_key_blocks(heads, kv_heads, hd, start, rows, q_f32, pad):
    """Edges of the 128-key blocks and 128-row tiles, heads that are no multiple of 64 depths, key ranges shared by the CTAs
    of a cluster (with and without a range for every CTA), query rows inside wider projected rows, and the f16 result."""
    rng = np.random.default_rng(heads * 7 + hd + start + rows)
    cache = sg.KvCache(heads, kv_heads, hd, start + rows + 200)
    cache._k.fill_(7.0)                                    # what lies past the last row must not count
    cache._v.fill_(-9.0)
    k16 = (rng.standard_normal((start + rows, kv_heads * hd)) * 0.7).astype(np.float16)
    v16 = rng.standard_normal((start + rows, kv_heads * hd)).astype(np.float16)
    cache.extend(torch.from_numpy(k16).cuda(), torch.from_numpy(v16).cuda())
    q32 = rng.standard_normal((rows, heads * hd)).astype(np.float32)
    if not q_f32:
        q32 = q32.astype(np.float16).astype(np.float32)
    q = torch.zeros((rows, heads * hd + pad), dtype=torch.float32 if q_f32 else torch.float16, device="cuda")
    q[:, :heads * hd] = torch.from_numpy(q32).cuda()
    out = torch.full((rows, heads * hd), 3.0, dtype=torch.float32, device="cuda")
    out16 = torch.full((rows, heads * hd), 3.0, dtype=torch.float16, device="cuda")
    cache._attend(q, heads * hd + pad, rows, out)
    cache._attend(q, heads * hd + pad, rows, out16)
    # the scalar statement in 64 bits (its f32 sums are within 1e-6 of it); the queries are rounded to f16 after the scale
    qh = (q32 * np.float32(cache.scale())).astype(np.float16).astype(np.float64).reshape(rows, kv_heads, heads // kv_heads, hd)
    kd, vd = (x.astype(np.float64).reshape(start + rows, kv_heads, hd) for x in (k16, v16))
    s = np.einsum("ikgd,tkd->kgit", qh, kd)
    s[:, :, np.arange(start + rows)[None, :] > start + np.arange(rows)[:, None]] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (np.einsum("kgit,tkd->ikgd", p, vd) / p.sum(-1).transpose(2, 0, 1)[..., None]).reshape(rows, heads * hd)
    # f32 scores of magnitude ~10 carry 1e-6, probabilities and their sums a few 2^-24 each
    assert max_rel(out.cpu().numpy(), want) <= 2e-5
    assert torch.equal(out16, out.half())
    assert sg.last_status() == 0


@pytest.mark.parametrize("heads,kv_heads,hd,start,rows", [(4, 2, 64, 100, 9), (8, 2, 128, 700, 1), (2, 2, 32, 0, 140)])
def test_non_finite_values_stay_with_the_rows_that_attend_to_them(heads, kv_heads, hd, start, rows):
    """An infinite value at one position: rows before it are as if it were not there, rows from it on have the infinity itself
    (not NaN) in its depth and their other depths untouched; a NaN key at the last position makes NaN of the last row alone."""
    rng = np.random.default_rng(heads + start)
    n = start + rows
    cache = sg.KvCache(heads, kv_heads, hd, n)
    k = torch.from_numpy((rng.standard_normal((n, kv_heads * hd)) * 0.5).astype(np.float16)).cuda()
    v = torch.from_numpy(rng.standard_normal((n, kv_heads * hd)).astype(np.float16)).cuda()
    q = torch.from_numpy(rng.standard_normal((rows, heads * hd)).astype(np.float16)).cuda()
    clean, bad = (torch.empty((rows, heads * hd), dtype=torch.float32, device="cuda") for _ in range(2))
    cache.extend(k, v)
    cache.attend_causal(q, rows, clean)
    at = start + rows // 2
    v[at, 5] = float("inf")                                    # KV head 0, depth 5
    cache.clear()
    cache.extend(k, v)
    cache.attend_causal(q, rows, bad)
    torch.cuda.synchronize()
    group = heads // kv_heads
    want = clean.clone()
    for h in range(group):
        want[at - start:, h * hd + 5] = float("inf")
    assert torch.equal(torch.isinf(bad), torch.isinf(want)) and not torch.isnan(bad).any()
    fin = torch.isfinite(want)
    assert max_rel(bad[fin].cpu().numpy(), want[fin].cpu().numpy()) <= 2e-5
    k[n - 1, 0] = float("nan")
    cache.clear()
    cache.extend(k, v)
    cache.attend_causal(q, rows, bad)
    torch.cuda.synchronize()
    assert torch.isnan(bad[rows - 1, :group * hd]).all() and not torch.isnan(bad[:rows - 1]).any() and not torch.isnan(bad[:, group * hd:]).any()
    assert sg.last_status() == 0


@pytest.mark.parametrize("heads,kv_heads,hd,start,rows,q_f32", [
    (4, 2, 64, 0, 1, False), (4, 2, 64, 63, 1, True), (8, 2, 128, 64, 3, False), (16, 1, 128, 511, 1, False), (6, 6, 40, 200, 2, True), (4, 4, 256, 130, 16, False),
    (2, 1, 72, 1000, 8, False), (8, 2, 128, 4090, 4, False), (3, 3, 32, 2050, 1, False), (32, 8, 128, 1023, 1, False)])
def test_decode_attention_runs_and_rows(heads, kv_heads, hd, start, rows, q_f32):
    """Up to 16 query rows per KV head: one run of keys and clusters of runs (some of them empty or past a row's last key),
    depths that are no multiple of 32 or 64, caches of one key."""
    rng = np.random.default_rng(heads + hd + start)
    n = start + rows
    cache = sg.KvCache(heads, kv_heads, hd, n + 100)
    cache._k.fill_(float("nan"))                           # what lies past the last row must not be read
    cache._v.fill_(float("nan"))
    k16 = (rng.standard_normal((n, kv_heads * hd)) * 0.7).astype(np.float16)
    v16 = rng.standard_normal((n, kv_heads * hd)).astype(np.float16)
    cache.extend(torch.from_numpy(k16).cuda(), torch.from_numpy(v16).cuda())
    q32 = rng.standard_normal((rows, heads * hd)).astype(np.float32)
    if not q_f32:
        q32 = q32.astype(np.float16).astype(np.float32)
    q = torch.from_numpy(q32).cuda().to(torch.float32 if q_f32 else torch.float16)
    out = torch.full((rows, heads * hd), 3.0, dtype=torch.float32, device="cuda")
    cache._attend(q, heads * hd, rows, out)
    qh = (q32 * np.float32(cache.scale())).astype(np.float16).astype(np.float64).reshape(rows, kv_heads, heads // kv_heads, hd)
    kd, vd = (x.astype(np.float64).reshape(n, kv_heads, hd) for x in (k16, v16))
    s = np.einsum("ikgd,tkd->kgit", qh, kd)
    s[:, :, np.arange(n)[None, :] > start + np.arange(rows)[:, None]] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (np.einsum("kgit,tkd->ikgd", p, vd) / p.sum(-1).transpose(2, 0, 1)[..., None]).reshape(rows, heads * hd)
    # f32 scores of magnitude ~10 carry 1e-6, probabilities and their sums a few 2^-24 each
    assert max_rel(out.cpu().numpy(), want) <= 2e-5
    assert sg.last_status() == 0


@pytest.mark.parametrize("rms", [True, False])
@pytest.mark.parametrize("d,heads,kv_heads,hd,rows", [(384, 6, 6, 64, 1), (256, 4, 2, 64, 2), (1152, 9, 3, 128, 1), (320, 5, 1, 64, 3)])
def test_layer_in_one_call_is_its_parts(rms, d, heads, kv_heads, hd, rows):
    """Block.accumulate as one library call (norms formed by the projections, keys and values written by the product) against
    the same layer run part by part: the same bits in the residual stream and in the caches."""
    rng = np.random.default_rng(d + rows)
    lin = lambda n, k: sg.Linear.quantize((rng.standard_normal((n, k)) * 0.05).astype(np.float32), sg.WeightLayout.OutIn, n, k)  # noqa: E731
    wt = lambda: rng.uniform(0.5, 1.5, d).astype(np.float32)  # noqa: E731
    norm = (lambda: sg.Norm.rms(wt(), 1e-5)) if rms else (lambda: sg.Norm.layer(wt(), wt() - 1, 1e-5))
    n1, n2 = norm(), norm()
    attn = sg.SelfAttention.new(lin((heads + 2 * kv_heads) * hd, d), lin(d, heads * hd), heads, kv_heads, hd)
    mlp = sg.Mlp.new(lin(2 * d, d), sg.Gate.Gelu, lin(d, 2 * d))
    block = sg.Block.new(n1, attn, n2, mlp)
    c1, c2 = block.cache(64), block.cache(64)
    x1 = torch.from_numpy(rng.standard_normal((rows, d)).astype(np.float32)).cuda()
    x2 = x1.clone()
    h = torch.empty((rows, d), dtype=torch.float16, device="cuda")
    for _ in range(3):
        block.accumulate(x1, c1, rows)
        n1.forward(x2, h)
        attn.accumulate(h, c2, x2, rows)
        n2.forward(x2, h)
        mlp.accumulate(h, x2, rows)
    torch.cuda.synchronize()
    assert torch.equal(x1, x2) and torch.equal(c1.keys(), c2.keys()) and torch.equal(c1.values(), c2.values())
    assert c1.len() == c2.len() == 3 * rows and sg.last_status() == 0


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("heads,kv_heads,hd,start,rows", [(4, 2, 64, 30, 1), (8, 2, 128, 700, 1), (4, 2, 64, 20, 40), (8, 1, 72, 300, 130)])
def test_results_go_to_buffers_off_the_16_byte_grid(heads, kv_heads, hd, start, rows, shift):
    """out may start at any element of a larger buffer (f32 and f16, one run and clusters of runs on both kernels): the bits of
    the aligned call, and nothing beside them is written."""
    rng = np.random.default_rng(heads + hd + shift)
    n, width = start + rows, heads * hd
    cache = sg.KvCache(heads, kv_heads, hd, n)
    cache.extend(*(torch.from_numpy(rng.standard_normal((n, kv_heads * hd)).astype(np.float16)).cuda() for _ in range(2)))
    q = torch.from_numpy(rng.standard_normal((rows, width)).astype(np.float16)).cuda()
    for dtype in (torch.float32, torch.float16):
        want = torch.empty((rows, width), dtype=dtype, device="cuda")
        cache._attend(q, width, rows, want)
        buf = torch.full((rows * width + 8,), 3.0, dtype=dtype, device="cuda")
        out = buf[shift:shift + rows * width]
        if rows == 1 and dtype == torch.float32:
            cache.attend(q, out)
        else:
            cache._attend(q, width, rows, out)
        torch.cuda.synchronize()
        assert torch.equal(out.view(rows, width), want)
        assert (buf[:shift] == 3.0).all() and (buf[shift + rows * width:] == 3.0).all()
    assert sg.last_status() == 0


@pytest.mark.parametrize("heads,kv_heads,hd,start,rows,kind", [
    (8, 8, 64, 192, 1, "nan"), (16, 8, 128, 448, 1, "nan"), (8, 8, 64, 192, 1, "inf"), (2, 1, 64, 0, 129, "nan"), (2, 1, 64, 0, 129, "inf"), (4, 2, 128, 256, 129, "nan")])
def test_a_nan_score_alone_in_its_run_of_keys_reaches_the_result(heads, kv_heads, hd, start, rows, kind):
    """The newest position's key makes a NaN score (a NaN, or infinities of both signs) and has a run of keys -- of the decode
    kernel, of a cluster's CTA -- to itself: the rows that attend to it are NaN, the others as without it."""
    rng = np.random.default_rng(heads + hd + start)
    n, at = start + rows, start + rows - 1
    k = torch.from_numpy((rng.standard_normal((n, kv_heads * hd)) * 0.5).astype(np.float16)).cuda()
    v = torch.from_numpy(rng.standard_normal((n, kv_heads * hd)).astype(np.float16)).cuda()
    q = torch.ones((rows, heads * hd), dtype=torch.float16, device="cuda")
    clean, bad = (torch.empty((rows, heads * hd), dtype=torch.float32, device="cuda") for _ in range(2))
    cache = sg.KvCache(heads, kv_heads, hd, n)
    cache.extend(k, v)
    cache.attend_causal(q, rows, clean)
    k[at, 0] = float(kind)                                     # KV head 0
    if kind == "inf":
        k[at, 1] = -float("inf")
    cache.clear()
    cache.extend(k, v)
    cache.attend_causal(q, rows, bad)
    torch.cuda.synchronize()
    hit = heads // kv_heads * hd
    assert torch.isnan(bad[rows - 1, :hit]).all()
    assert torch.equal(bad[rows - 1, hit:], clean[rows - 1, hit:]) and torch.equal(bad[:rows - 1], clean[:rows - 1])
    assert sg.last_status() == 0


@pytest.mark.parametrize("out16", [False, True])
@pytest.mark.parametrize("heads,kv_heads,hd,start,rows", [(4, 2, 64, 40, 1), (16, 8, 128, 900, 1), (8, 2, 72, 300, 3), (32, 8, 128, 512, 512), (4, 2, 256, 0, 140), (4, 4, 40, 0, 130)])
def test_an_early_non_finite_value_costs_a_pass_and_not_seconds(heads, kv_heads, hd, start, rows, out16):
    """An infinity of either sign and a NaN among the values of position 0 (KV head 0), an infinity among the last one's: every
    row of that head's group is formed again, exactly as the 64-bit statement has it, in a time of the kernel's own order."""
    rng = np.random.default_rng(heads + hd + rows)
    n, group = start + rows, heads // kv_heads
    k = torch.from_numpy((rng.standard_normal((n, kv_heads * hd)) * 0.5).astype(np.float16)).cuda()
    v = torch.from_numpy(rng.standard_normal((n, kv_heads * hd)).astype(np.float16)).cuda()
    v[0, 3], v[0, hd - 1], v[0, hd // 2], v[n - 1, 9] = float("inf"), -float("inf"), float("nan"), float("inf")
    q = torch.from_numpy(rng.standard_normal((rows, heads * hd)).astype(np.float16)).cuda()
    out = torch.empty((rows, heads * hd), dtype=torch.float16 if out16 else torch.float32, device="cuda")
    cache = sg.KvCache(heads, kv_heads, hd, n)
    cache.extend(k, v)
    cache._attend(q, heads * hd, rows, out)
    torch.cuda.synchronize()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record()
    cache._attend(q, heads * hd, rows, out)
    ev[1].record()
    torch.cuda.synchronize()
    qh = (q.float() * np.float32(cache.scale())).half().double().view(rows, kv_heads, group, hd)
    s = torch.einsum("ikgd,tkd->kgit", qh, k.double().view(n, kv_heads, hd))
    s.masked_fill_(torch.arange(n, device="cuda")[None, :] > start + torch.arange(rows, device="cuda")[:, None], -float("inf"))
    p = torch.softmax(s, -1)
    fin = torch.nan_to_num(v.double(), nan=0.0, posinf=0.0, neginf=0.0)
    want = torch.einsum("kgit,tkd->ikgd", p, fin.view(n, kv_heads, hd)).reshape(rows, group * kv_heads, hd)
    want[:, :group, 3], want[:, :group, hd - 1], want[:, :group, hd // 2] = float("inf"), -float("inf"), float("nan")
    want[rows - 1, :group, 9] = float("inf")
    want, got = want.reshape(rows, heads * hd), out.double()
    ok = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    # f32 sums as elsewhere in this file; half a place of the f16 store on top
    assert ((got - want).abs()[ok] / (1 + want.abs()[ok])).max() <= (2e-5 + 2.0 ** -11 if out16 else 2e-5)
    assert ev[0].elapsed_time(ev[1]) < 25.0                   # (measured 1.7 at the largest; a thread per eight depths took hundreds)
    assert sg.last_status() == 0


@pytest.mark.parametrize("q_scale", [1.0, 6.0])
@pytest.mark.parametrize("heads,kv_heads,hd,start,rows", [(16, 2, 64, 300, 300), (16, 4, 128, 4000, 1), (12, 12, 32, 64, 100), (8, 2, 128, 700, 130)])
def test_no_further_from_64_bits_than_the_scalar_statement(heads, kv_heads, hd, start, rows, q_scale):
    """The error of the f32 result against the statement in 64 bits, beside the error of the scalar f32 statement itself, over
    flat and sharp distributions: probabilities in two parts and tensor-core sums lose nothing against f32 in key order."""
    n, err, err_scalar = start + rows, 0.0, 0.0
    for seed in range(3):
        rng = np.random.default_rng(heads + hd + start + 1000 * seed)
        k16, v16 = (rng.standard_normal((n, kv_heads * hd)).astype(np.float16) for _ in range(2))
        q32 = (rng.standard_normal((rows, heads * hd)) * q_scale).astype(np.float16).astype(np.float32)
        cache = sg.KvCache(heads, kv_heads, hd, n)
        cache.extend(torch.from_numpy(k16).cuda(), torch.from_numpy(v16).cuda())
        out = torch.empty((rows, heads * hd), dtype=torch.float32, device="cuda")
        cache.attend_causal(torch.from_numpy(q32.astype(np.float16)).cuda(), rows, out)
        scalar = orc.attention_kv_causal(q32, k16.view(np.uint16), v16.view(np.uint16), start, rows, heads, kv_heads, hd, cache.scale())
        qh = (q32 * np.float32(cache.scale())).astype(np.float16).astype(np.float64).reshape(rows, kv_heads, heads // kv_heads, hd)
        kd, vd = (x.astype(np.float64).reshape(n, kv_heads, hd) for x in (k16, v16))
        s = np.einsum("ikgd,tkd->kgit", qh, kd)
        s[:, :, np.arange(n)[None, :] > start + np.arange(rows)[:, None]] = -np.inf
        p = np.exp(s - s.max(-1, keepdims=True))
        want = (np.einsum("kgit,tkd->ikgd", p, vd) / p.sum(-1).transpose(2, 0, 1)[..., None]).reshape(rows, heads * hd)
        err += float(((out.cpu().numpy() - want) ** 2).sum())
        err_scalar += float(((np.asarray(scalar).reshape(want.shape) - want) ** 2).sum())
    # (a tenth for the draw: two orders of the same f32 sums differ by that much)
    assert err ** 0.5 <= 1.1 * err_scalar ** 0.5 and sg.last_status() == 0


def test_more_query_rows_of_a_head_than_one_grid_has_tiles():
    """8192 heads on one KV head x 1100 rows: 70400 tiles of 128 query rows, past the 65535 of a grid's dimension."""
    heads, hd, rows = 8192, 8, 1100
    g = torch.Generator(device="cuda").manual_seed(3)
    k, v = (torch.randn(rows, hd, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(rows, heads * hd, generator=g, device="cuda").half()
    out = torch.full((rows, heads * hd), 3.0, dtype=torch.float32, device="cuda")
    cache = sg.KvCache(heads, 1, hd, rows)
    cache.extend(k, v)
    cache.attend_causal(q, rows, out)
    for i in (0, 1, 511, 1022, 1023, 1024, 1025, rows - 1):    # 65535 tiles end in row 1023
        qh = (q[i].float() * np.float32(cache.scale())).half().double().view(heads, hd)
        p = torch.softmax(qh @ k[:i + 1].double().T, -1)
        want = (p @ v[:i + 1].double()).reshape(-1)
        assert ((out[i].double() - want).abs() / (1 + want.abs())).max() <= 2e-5
    assert not (out == 3.0).all(1).any() and sg.last_status() == 0
