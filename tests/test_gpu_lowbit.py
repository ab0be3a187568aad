"""2-bit / 1-bit int8-activation kernels on the GPU: BIT-EXACT against the CPU
oracle (quantize_row + reference, src/kernels/lowbit/matmul.rs:354-398) --
int8 activation codes, per-block activation scales, int32 block sums and the f16
output, for the reference's own shape / block / codebook / layout grid
(src/kernels/lowbit/matmul.rs:419-494), through the C ABI."""
import os

import numpy as np
import pytest
import torch

import oracle as orc
import sme_gemm_b200 as sg
from gpu_util import bits_of, f16_bits_dev
from refgen import Lcg, data

pytestmark = pytest.mark.gpu

SHAPES = [(1, 64, 256), (1, 65, 37), (1, 1, 1), (2, 200, 300), (3, 64, 16), (5, 130, 513), (6, 192, 256),
          (7, 100, 64), (12, 70, 200), (1, 2048, 1024), (4, 1536, 512), (9, 1024, 384)]
BOOKS = [[-1, 0, 1, 0], [-2, -1, 1, 2], [-128, 127, 3, -7]]


def _canon16(bits):
    """f16 bit patterns with every NaN mapped to one pattern (NaN payloads are not part of the contract)."""
    b = np.array(bits, np.uint16, copy=True)
    b[(b & 0x7fff) > 0x7c00] = 0x7e00
    return b


def _canon32(x):
    b = np.array(x, np.float32, copy=True).view(np.uint32)
    b[(b & 0x7fffffff) > 0x7f800000] = 0x7fc00000
    return b


def check_bits(w, kind, wbits, layout, scales, book, n, k, block, m, a_bits, what):
    c, q, sa, sums = sg.matmul_lowbit_debug(f16_bits_dev(a_bits).reshape(m, k), w, m)
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    wc, wq, wsa, wsums = orc.lowbit_matmul(a_bits, kind, wbits, layout, scales, book, n, k, block, m, debug=True)
    assert np.array_equal(q.cpu().numpy(), wq), f"{what}: int8 activation codes differ"
    assert np.array_equal(_canon32(sa.cpu().numpy()), _canon32(wsa)), f"{what}: activation scales differ"
    assert np.array_equal(sums.cpu().numpy(), wsums), f"{what}: int32 block sums differ"
    got, wc = _canon16(bits_of(c)), _canon16(wc)
    bad = np.nonzero(got != wc)
    assert bad[0].size == 0, f"{what}: {bad[0].size} of {got.size} f16 outputs differ, first at {bad[0][0]},{bad[1][0]}"
    # the plain entry point gives the same bits
    c2 = torch.full((m, n), 9.0, dtype=torch.float16, device="cuda")
    (sg.matmul_q2 if kind == 2 else sg.matmul_q1)(f16_bits_dev(a_bits), w, c2, m)
    assert np.array_equal(_canon16(bits_of(c2)), wc), f"{what}: plain call differs"


@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_kernels_match_reference_bits(si):
    m, n, k = SHAPES[si]
    for bi, block in enumerate([16, 64, 128, 4096]):
        nbk = -(-k // block)
        scales = orc.f32_to_f16_bits(data(si + 7, n * nbk).astype(np.float32) * np.float32(1e-3) - np.float32(0.1))
        a_bits = orc.f32_to_f16_bits((data(si + 99, m * k).astype(np.float32) - np.float32(128.0)) / np.float32(37.0))
        book = BOOKS[(si + bi) % 3]
        codes = data(si * 31 + bi, (k * n + 3) // 4)
        w2 = sg.Q2Weights.new(codes, scales, n, k, sg.Q2Params(block).with_codebook(book))
        check_bits(w2, 2, codes, 1, scales, book, n, k, block, m, a_bits, f"q2 {m}x{n}x{k} block {block} {book}")
        signs = data(si * 17 + bi, (k * n + 7) // 8)
        for layout in (0, 1):
            w1 = sg.Q1Weights.new(signs, scales, sg.WeightLayout(layout), n, k, block)
            check_bits(w1, 1, signs, layout, scales, None, n, k, block, m, a_bits, f"q1 {m}x{n}x{k} block {block} layout {layout}")


def test_results_do_not_depend_on_m():
    """"Results do not depend on m" (src/kernels/lowbit/matmul.rs:24-25): row i of an
    m-row call equals the one-row call on that row, bit for bit."""
    n, k, block = 200, 1024, 128
    rng = np.random.default_rng(2)
    codes = rng.integers(0, 256, (k * n + 3) // 4).astype(np.uint8)
    scales = orc.f32_to_f16_bits(rng.uniform(0.01, 0.05, n * (k // block)).astype(np.float32))
    w = sg.Q2Weights.new(codes, scales, n, k, sg.Q2Params(block))
    a = torch.from_numpy(rng.standard_normal((19, k)).astype(np.float16)).cuda()
    c = torch.zeros((19, n), dtype=torch.float16, device="cuda")
    sg.matmul_q2(a, w, c, 19)
    for i in (0, 7, 8, 18):
        ci = torch.zeros((1, n), dtype=torch.float16, device="cuda")
        sg.matmul_q2(a[i:i + 1].contiguous(), w, ci, 1)
        assert torch.equal(ci.view(torch.int16)[0], c.view(torch.int16)[i])


def test_nan_and_inf_activations_follow_quantize_row():
    n, k, block = 64, 256, 64
    rng = np.random.default_rng(3)
    signs = rng.integers(0, 256, (k * n + 7) // 8).astype(np.uint8)
    scales = orc.f32_to_f16_bits(rng.uniform(0.005, 0.03, n * (k // block)).astype(np.float32))
    a = rng.standard_normal((2, k)).astype(np.float16)
    a[0, 5] = np.nan
    a[1, 70] = np.inf
    w = sg.Q1Weights.new(signs, scales, sg.WeightLayout.OutIn, n, k, block)
    check_bits(w, 1, signs, 0, scales, None, n, k, block, 2, a.view(np.uint16), "nan/inf rows")


def test_epilogue_on_the_f16_rounded_product_is_bit_exact():
    """config 3's graph: mul_col(s).add_col(b), evaluated as apply_ep_scalar does
    (src/kernels/lowbit/matmul.rs:335-336, src/exec/scalar.rs:125-140); plus a bias /
    row scale / trailing gelu graph within 1e-2 (tests/correctness/q2.rs:83-106)."""
    m, n, k, block = 8, 300, 512, 128
    rng = np.random.default_rng(4)
    signs = rng.integers(0, 256, (k * n + 7) // 8).astype(np.uint8)
    scales = orc.f32_to_f16_bits(rng.uniform(0.005, 0.03, n * (k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal((m, k)).astype(np.float32))
    s_bits = orc.f32_to_f16_bits(rng.uniform(0.5, 1.5, n).astype(np.float32))
    b_bits = orc.f32_to_f16_bits((rng.standard_normal(n) * 0.1).astype(np.float32))
    w = sg.Q1Weights.new(signs, scales, sg.WeightLayout.InOut, n, k, block)
    c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
    sg.matmul_q1_ep(f16_bits_dev(a_bits), w, c, m, sg.Epilogue().mul_col(f16_bits_dev(s_bits)).add_col(f16_bits_dev(b_bits)))
    want = orc.lowbit_matmul(a_bits, 1, signs, 1, scales, None, n, k, block, m)
    want = orc.apply_ep(want, m, n, orc.Nodes([(5, 0, 0.0, s_bits, 0), (4, 0, 0.0, b_bits, 0)]))
    assert np.array_equal(bits_of(c), want)
    row = orc.f32_to_f16_bits(rng.uniform(0.5, 1.5, m).astype(np.float32))
    sg.matmul_q1_ep(f16_bits_dev(a_bits), w, c, m,
                    sg.Epilogue().add_col(f16_bits_dev(b_bits)).mul_row(f16_bits_dev(row)).gelu())
    want = orc.lowbit_matmul(a_bits, 1, signs, 1, scales, None, n, k, block, m)
    want = orc.apply_ep(want, m, n, orc.Nodes([(4, 0, 0.0, b_bits, 0), (3, 0, 0.0, row, 0), (8, 2, 0.0, None, 0)]))
    assert np.max(np.abs(c.float().cpu().numpy() - orc.f16_bits_to_f32(want))) <= 1e-2


def test_config2_ternary_gemv_full_size():
    """M=1, K=4096, N=11008, codes i.i.d. in {-1,0,+1}, block 256, scales U(0.01,0.05)."""
    m, n, k, block = 1, 11008, 4096, 256
    rng = np.random.default_rng(12)
    two = rng.integers(0, 3, k * n).astype(np.uint8)
    codes = (two[0::4] | (two[1::4] << 2) | (two[2::4] << 4) | (two[3::4] << 6)).astype(np.uint8)
    scales = orc.f32_to_f16_bits(rng.uniform(0.01, 0.05, n * (k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal((m, k)).astype(np.float32))
    w = sg.Q2Weights.new(codes, scales, n, k)
    check_bits(w, 2, codes, 1, scales, BOOKS[0], n, k, block, m, a_bits, "config 2")


def test_config3_one_bit_batch_full_size():
    """M=8, K=4096, N=14336, Bernoulli(0.5) signs, block 128, mul_col(s).add_col(b)."""
    m, n, k, block = 8, 14336, 4096, 128
    rng = np.random.default_rng(13)
    signs = rng.integers(0, 256, (k * n) // 8).astype(np.uint8)
    scales = orc.f32_to_f16_bits(rng.uniform(0.005, 0.03, n * (k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal((m, k)).astype(np.float32))
    w = sg.Q1Weights.new(signs, scales, sg.WeightLayout.OutIn, n, k, block)
    check_bits(w, 1, signs, 0, scales, None, n, k, block, m, a_bits, "config 3")
    s_bits = orc.f32_to_f16_bits(rng.uniform(0.5, 1.5, n).astype(np.float32))
    b_bits = orc.f32_to_f16_bits((rng.standard_normal(n) * 0.1).astype(np.float32))
    c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
    sg.matmul_q1_ep(f16_bits_dev(a_bits), w, c, m, sg.Epilogue().mul_col(f16_bits_dev(s_bits)).add_col(f16_bits_dev(b_bits)))
    want = orc.apply_ep(orc.lowbit_matmul(a_bits, 1, signs, 0, scales, None, n, k, block, m), m, n,
                        orc.Nodes([(5, 0, 0.0, s_bits, 0), (4, 0, 0.0, b_bits, 0)]))
    assert np.array_equal(bits_of(c), want)


def test_host_and_drop_in_entries_and_pack_roundtrip():
    m, n, k, block = 4, 130, 300, 64
    rng = np.random.default_rng(6)
    codes = rng.integers(0, 256, (k * n + 3) // 4).astype(np.uint8)
    codes[-1] &= (1 << (2 * ((k * n) % 4 or 4))) - 1
    nbk = -(-k // block)
    scales = orc.f32_to_f16_bits(rng.uniform(0.01, 0.05, n * nbk).astype(np.float32))
    a = rng.standard_normal((m, k)).astype(np.float16)
    book = BOOKS[1]
    want = orc.lowbit_matmul(a, 2, codes, 1, scales, book, n, k, block, m)
    w = sg.Q2Weights.new(codes, scales, n, k, sg.Q2Params(block).with_codebook(book))
    c = np.zeros((m, n), np.float16)
    sg.matmul_q2(a, w, c, m)
    assert np.array_equal(c.view(np.uint16), want)
    back, sback = w.unpack()
    assert np.array_equal(back, codes) and np.array_equal(sback, scales)
    # the reference's band-major arrays through the reference's own symbols
    packed, sc = orc.q2_pack_band(codes, scales, n, k, block)
    L = sg.lib()
    cb = np.asarray(book, np.int8)
    c2 = np.zeros((m, n), np.uint16)
    assert L.gemm_sme_f16_q2(m, n, k, c2.ctypes.data, a.ctypes.data, packed.ctypes.data, sc.ctypes.data, cb.ctypes.data, block, None) == 0
    assert np.array_equal(c2, want)
    L.smeg_forget(packed.ctypes.data)
    signs = rng.integers(0, 256, (k * n + 7) // 8).astype(np.uint8)
    want1 = orc.lowbit_matmul(a, 1, signs, 0, scales, None, n, k, block, m)
    packed1, sc1 = orc.q1_pack_band(signs, 0, scales, n, k, block)
    c3 = np.zeros((m, n), np.uint16)
    assert L.gemm_sme_f16_q1(m, n, k, c3.ctypes.data, a.ctypes.data, packed1.ctypes.data, sc1.ctypes.data, block, None) == 0
    assert np.array_equal(c3, want1)
    L.smeg_forget(packed1.ctypes.data)


def test_q1_interleave_keeps_every_column():
    """src/kernels/lowbit/q1.rs:298-319."""
    n, k, block = 70, 300, 64
    rng = np.random.default_rng(8)
    wg = rng.standard_normal(n * k).astype(np.float32)
    wu = rng.standard_normal(n * k).astype(np.float32)
    g = sg.Q1Weights.quantize(wg, sg.WeightLayout.OutIn, n, k, block)
    u = sg.Q1Weights.quantize(wu, sg.WeightLayout.OutIn, n, k, block)
    both = sg.Q1Weights.interleave(g, u)
    a = torch.from_numpy(rng.standard_normal((2, k)).astype(np.float16)).cuda()
    cg, cu = (torch.zeros((2, n), dtype=torch.float16, device="cuda") for _ in range(2))
    cb = torch.zeros((2, 2 * n), dtype=torch.float16, device="cuda")
    sg.matmul_q1(a, g, cg, 2); sg.matmul_q1(a, u, cu, 2); sg.matmul_q1(a, both, cb, 2)
    col = 0
    for c0 in range(0, n, 32):
        w = min(32, n - c0)
        assert torch.equal(cb[:, col:col + w], cg[:, c0:c0 + w]); col += w
        assert torch.equal(cb[:, col:col + w], cu[:, c0:c0 + w]); col += w


@pytest.mark.parametrize("m,n,k", [(65, 70, 512), (200, 300, 1024), (130, 1000, 320)])
def test_many_rows_on_the_tensor_cores_are_the_reference_bits(m, n, k):
    """Seventeen rows and up run on tcgen05 (64-row tiles, or 128-row tiles with the totals in tensor memory where a
    K-block is 64 to 256 deep): the plain entry points against the scalar statement, ragged column tiles included."""
    rng = np.random.default_rng(m + n)
    a_bits = orc.f32_to_f16_bits(rng.standard_normal((m, k)).astype(np.float32))
    for block in (16, 64, 128, 256, 1024):
        nbk = -(-k // block)
        scales = orc.f32_to_f16_bits(rng.uniform(0.01, 0.05, n * nbk).astype(np.float32))
        codes = rng.integers(0, 256, (k * n + 3) // 4).astype(np.uint8)
        book = BOOKS[(block // 16) % 3]
        w2 = sg.Q2Weights.new(codes, scales, n, k, sg.Q2Params(block).with_codebook(book))
        c = torch.full((m, n), 9.0, dtype=torch.float16, device="cuda")
        sg.matmul_q2(f16_bits_dev(a_bits), w2, c, m)
        want = orc.lowbit_matmul(a_bits, 2, codes, 1, scales, book, n, k, block, m)
        assert np.array_equal(_canon16(bits_of(c)), _canon16(want)), f"q2 {m}x{n}x{k} block {block}"
        signs = rng.integers(0, 256, (k * n + 7) // 8).astype(np.uint8)
        w1 = sg.Q1Weights.new(signs, scales, sg.WeightLayout.OutIn, n, k, block)
        sg.matmul_q1(f16_bits_dev(a_bits), w1, c, m)
        want = orc.lowbit_matmul(a_bits, 1, signs, 0, scales, None, n, k, block, m)
        assert np.array_equal(_canon16(bits_of(c)), _canon16(want)), f"q1 {m}x{n}x{k} block {block}"
    assert sg.last_status() == 0


@pytest.mark.parametrize("m,n,k,block", [(17, 129, 256, 16), (33, 300, 1000, 32), (65, 130, 640, 64), (97, 128, 1501, 128), (129, 200, 700, 256),
                                         (300, 70, 384, 128), (32, 2000, 130, 256), (220, 1100, 2048, 64)])
@pytest.mark.parametrize("kind", [1, 2])
def test_row_tiles_of_the_block_kernel(kind, m, n, k, block):
    """Every row tile (32 to 128 rows) with rows and columns missing, accumulators of one stage, of two and several to a stage,
    depths that end inside a stage; rows of zeros, infinities and NaN among the others."""
    rng = np.random.default_rng(m + n + k + kind)
    nbk = -(-k // block)
    scales = orc.f32_to_f16_bits((rng.standard_normal(n * nbk) * 0.02).astype(np.float32))
    scales[:3] = (0x7c00, 0x0001, 0x8000)                        # an infinite, a subnormal and a negative zero scale
    a32 = rng.standard_normal((m, k)).astype(np.float32) * 3
    a32[1], a32[3, k // 2], a32[5, 0], a32[m - 1, k - 1] = 0.0, np.nan, np.inf, -65504.0
    a_bits = orc.f32_to_f16_bits(a32)
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8).astype(np.uint8)
    book = BOOKS[m % 3]
    w = (sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(book)) if kind == 2
         else sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block))
    c = torch.full((m, n), 9.0, dtype=torch.float16, device="cuda")
    (sg.matmul_q2 if kind == 2 else sg.matmul_q1)(f16_bits_dev(a_bits), w, c, m)
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    want = orc.lowbit_matmul(a_bits, kind, wbits, 1 if kind == 2 else 0, scales, book if kind == 2 else None, n, k, block, m)
    want = want[0] if isinstance(want, tuple) else want
    assert np.array_equal(_canon16(bits_of(c)).reshape(-1), _canon16(want).reshape(-1))


# The kernel of one to sixteen rows: depths in one part, in four and in eight, K-blocks longer than a part's share, a depth that
# ends inside a unit, a part without a whole K-block, more column groups than a round of a CTA's warps, rows past a tile of eight, and
# more values than a CTA quantises for itself.
@pytest.mark.parametrize("m,n,k,block", [(1, 40, 3000, 32), (2, 300, 12500, 128), (3, 70, 1000, 1024), (5, 33, 8200, 64), (8, 2400, 700, 256),
                                         (9, 100, 4500, 128), (11, 64, 2049, 512), (16, 50, 2600, 128), (1, 40000, 256, 128), (16, 37900, 160, 32)])
@pytest.mark.parametrize("kind", [1, 2])
def test_parts_and_tiles_of_the_kernel_for_few_rows(kind, m, n, k, block):
    rng = np.random.default_rng(m * 1000 + k)
    scales = orc.f32_to_f16_bits(rng.uniform(-0.05, 0.05, n * -(-k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32))
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8).astype(np.uint8)
    if kind == 2:
        w = sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(BOOKS[2]))
        check_bits(w, 2, wbits, 1, scales, BOOKS[2], n, k, block, m, a_bits, "q2")
    else:
        w = sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block)
        check_bits(w, 1, wbits, 0, scales, None, n, k, block, m, a_bits, "q1")


@pytest.mark.parametrize("m", [1, 6, 12])
def test_resolved_graphs_of_the_kernel_for_few_rows(m):
    """Scalars and column vectors without an activation, node by node on the f16 product: the interpreter's bits (numpy's f32)."""
    n, k = 131, 512
    rng = np.random.default_rng(m)
    scales = orc.f32_to_f16_bits(rng.uniform(0.01, 0.05, n * 4).astype(np.float32))
    w = sg.Q1Weights.new(rng.integers(0, 256, k * n // 8).astype(np.uint8), scales, sg.WeightLayout.OutIn, n, k, 128)
    a = f16_bits_dev(orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32)))
    v = [rng.standard_normal(n).astype(np.float16) for _ in range(4)]
    d = [torch.from_numpy(x).cuda() for x in v]
    f = [x.astype(np.float32) for x in v]
    plain = torch.empty((m, n), dtype=torch.float16, device="cuda")
    sg.matmul_q1(a, w, plain, m)
    x = plain.cpu().numpy().astype(np.float32)
    for ep, want in ((sg.Epilogue().mul_col(d[0]).add_col(d[1]).sub_col(d[2]).max_col(d[3]), np.maximum((x * f[0] + f[1]) - f[2], f[3])),
                     (sg.Epilogue().add_scalar(0.5).mul_scalar(3.0).sub_scalar(0.25).min(1.5), np.minimum((x + np.float32(0.5)) * 3 - np.float32(0.25), np.float32(1.5))),
                     (sg.Epilogue().max(-0.5).min_col(d[0]), np.minimum(np.maximum(x, np.float32(-0.5)), f[0]))):
        c = torch.empty_like(plain)
        sg.matmul_q1_ep(a, w, c, m, ep)
        assert np.array_equal(c.cpu().numpy().view(np.uint16), want.astype(np.float16).view(np.uint16))


# Depths whose parts have room only because no more is laid out than is at work (one and two column groups a CTA), for one and
# two tiles of rows; the last ones are left to other kernels (one part of sixteen, one group a CTA).
@pytest.mark.parametrize("m,n,k,block", [(1, 70, 14336, 64), (1, 4800, 8192, 32), (2, 64, 16384, 128), (7, 70, 8192, 64), (6, 4800, 4096, 32), (13, 33, 8192, 256),
                                         (10, 2500, 3000, 64), (16, 70, 4096, 64), (16, 40, 8192, 64), (12, 40, 16384, 512)])
@pytest.mark.parametrize("kind", [1, 2])
def test_deep_parts_of_the_kernel_for_few_rows(kind, m, n, k, block):
    rng = np.random.default_rng(m * 1000 + k)
    scales = orc.f32_to_f16_bits(rng.uniform(-0.05, 0.05, n * -(-k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32))
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8).astype(np.uint8)
    if kind == 2:
        w = sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(BOOKS[1]))
        check_bits(w, 2, wbits, 1, scales, BOOKS[1], n, k, block, m, a_bits, "q2")
    else:
        w = sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block)
        check_bits(w, 1, wbits, 0, scales, None, n, k, block, m, a_bits, "q1")


# Either side of the lines between the kernel for few rows and the one for one and two (whose long K-blocks are longer than a unit), and
# between quantising in the CTAs and in front for K-blocks above 256.
@pytest.mark.parametrize("m,n,k,block", [(1, 100, 2048, 256), (2, 100, 2050, 256), (1, 64, 257, 64), (2, 40, 1024, 128), (1, 70, 12288, 512), (1, 2400, 3000, 1024), (2, 40, 6144, 4096),
                                         (2, 40, 6400, 1024), (8, 64, 4096, 512), (9, 64, 3000, 512), (16, 40, 2048, 2048), (3, 40, 4200, 8192)])
@pytest.mark.parametrize("kind", [1, 2])
def test_lines_of_the_dispatch_at_few_rows(kind, m, n, k, block):
    rng = np.random.default_rng(m * 1000 + k)
    scales = orc.f32_to_f16_bits(rng.uniform(-0.05, 0.05, n * -(-k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32))
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8).astype(np.uint8)
    if kind == 2:
        w = sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(BOOKS[2]))
        check_bits(w, 2, wbits, 1, scales, BOOKS[2], n, k, block, m, a_bits, "q2")
    else:
        w = sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block)
        check_bits(w, 1, wbits, 0, scales, None, n, k, block, m, a_bits, "q1")


_COUNT_NODES = r"""
import numpy as np, torch
import sme_gemm_b200 as sg
from cuda.bindings import runtime as rt
rng = np.random.default_rng(0)
n, k = 64, 512
w = sg.Q1Weights.new(rng.integers(0, 256, n * k // 8).astype(np.uint8), np.full(n * k // 128, 0.01, np.float16).view(np.uint16), sg.WeightLayout.OutIn, n, k, 128)
s = torch.cuda.Stream()
for m in (4, 7, 9):
    a = torch.ones((m, k), dtype=torch.float16, device="cuda")
    c = torch.empty((m, n), dtype=torch.float16, device="cuda")
    with torch.cuda.stream(s):
        sg.matmul_q1(a, w, c, m)
        s.synchronize()
        assert rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
        sg.matmul_q1(a, w, c, m)
        err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
    assert err == 0
    err, _, count = rt.cudaGraphGetNodes(graph)
    err, nodes, count = rt.cudaGraphGetNodes(graph, count)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes[:count]]
    print(m, sum(x == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for x in kinds))
    rt.cudaGraphDestroy(graph)
"""


@pytest.mark.parametrize("knob,launches", [(None, {4: 1, 7: 1, 9: 1}), ("8", {4: 1, 7: 1, 9: 2})])
def test_rows_from_which_tcgen05_takes_a_call(knob, launches):
    """SMEG_LOWBIT_TC_MIN_ROWS holds for calls of any size: from its rows on a call is the quantisation and the tcgen05 kernel, two
    launches, where the kernel for few rows is one."""
    import subprocess
    import sys
    env = {x: v for x, v in os.environ.items() if x != "SMEG_LOWBIT_TC_MIN_ROWS"}
    if knob:
        env["SMEG_LOWBIT_TC_MIN_ROWS"] = knob
    env["PYTHONPATH"] = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _COUNT_NODES], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert dict(map(int, line.split()) for line in r.stdout.splitlines()) == launches


# Five to sixteen rows whose codes do not fit a CTA, or would be one part of one group's depth: the kernel on f16 instructions, one and
# two tiles of rows, K-blocks of a unit and longer and (two tiles, 1-bit) shorter ones; the last is left to the staged kernel.
@pytest.mark.parametrize("kind,m,n,k,block", [(1, 8, 40, 28672, 256), (2, 8, 40, 28672, 256), (2, 5, 24, 60000, 1024), (1, 12, 40, 16384, 512), (2, 12, 40, 16384, 512),
                                              (2, 12, 33, 16000, 256), (1, 9, 40, 15360, 128), (1, 16, 40, 8192, 64), (2, 16, 24, 8192, 32)])
def test_deep_rows_of_the_kernels_behind(kind, m, n, k, block):
    rng = np.random.default_rng(m * 1000 + k)
    scales = orc.f32_to_f16_bits(rng.uniform(-0.05, 0.05, n * -(-k // block)).astype(np.float32))
    a_bits = orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32))
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8).astype(np.uint8)
    if kind == 2:
        w = sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(BOOKS[2]))
        check_bits(w, 2, wbits, 1, scales, BOOKS[2], n, k, block, m, a_bits, "q2")
    else:
        w = sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block)
        check_bits(w, 1, wbits, 0, scales, None, n, k, block, m, a_bits, "q1")


@pytest.mark.parametrize("kind,m,k,block", [(1, 5, 6464, 32), (2, 5, 6560, 32), (2, 9, 7520, 64)])
def test_wide_matrices_of_the_kernel_behind(kind, m, k, block):
    """K-blocks shorter than a unit reach the kernel on f16 instructions where a CTA has sixteen groups whose scale rows leave its codes
    no room: each row's bits are those of a call of that row alone, which runs on the kernel for few rows."""
    n = 35600
    rng = np.random.default_rng(k)
    scales = orc.f32_to_f16_bits(rng.uniform(-0.05, 0.05, n * -(-k // block)).astype(np.float32))
    wbits = rng.integers(0, 256, (k * n * kind + 7) // 8, dtype=np.uint8)
    if kind == 2:
        w, f = sg.Q2Weights.new(wbits, scales, n, k, sg.Q2Params(block).with_codebook(BOOKS[1])), sg.matmul_q2
    else:
        w, f = sg.Q1Weights.new(wbits, scales, sg.WeightLayout.OutIn, n, k, block), sg.matmul_q1
    a = f16_bits_dev(orc.f32_to_f16_bits(rng.standard_normal(m * k).astype(np.float32))).reshape(m, k)
    c, one = torch.zeros((m, n), dtype=torch.float16, device="cuda"), torch.zeros((1, n), dtype=torch.float16, device="cuda")
    f(a, w, c, m)
    for r in range(m):
        f(a[r:r + 1].contiguous(), w, one, 1)
        assert np.array_equal(_canon16(bits_of(c[r:r + 1])), _canon16(bits_of(one)))
