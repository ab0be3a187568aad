"""Prefill calls on the GPU against the CPU oracle, through the C ABI.

Above 16 rows a call runs on the tensor-core kernel (tcgen05 / TMEM) or, on small matrices, on the
warp-level one: tests of the former say so (takes_gemm).  Tolerance as
for the decode path: max |g-w|/(1+|w|) <= 1e-2 against the oracle (same f32
accumulation over the same rounded weights; only the summation order differs)."""
import numpy as np
import pytest
import torch

import oracle as orc
import sme_gemm_b200 as sg
from gpu_util import bf16_bits_dev, bits_of, f16_bits_dev, max_rel, q4_logical, takes_gemm

pytestmark = pytest.mark.gpu
TOL = 1e-2
# bf16 through an epilogue: the product is rounded to bf16 before the graph (as the reference does), a different
# summation order can flip that rounding by one ulp (2^-8 relative), and the activation carries it to at most two ulps
# of the result: 2e-2 on the 1/(1+|w|) metric.  Still far inside the reference's own sqrt(k)-scaled bound
# (max(1e-2, 1e-2*sqrt(k)/4) = 0.16 at k = 4096).
TOL_BF16_EP = 2e-2


def run(m, n, k, block, bf16, seed=0, ep=None, sample_rows=None):
    rng = np.random.default_rng(seed + m * 131 + n * 17 + k)
    q, s = q4_logical(rng, n, k, block)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(block))
    a32 = rng.standard_normal((m, k)).astype(np.float32)
    a_bits = orc.f32_to_bf16_bits(a32) if bf16 else orc.f32_to_f16_bits(a32)
    to_dev = bf16_bits_dev if bf16 else f16_bits_dev
    dt = "bf16" if bf16 else "f16"
    epi, nodes = None, None
    if ep == "cfg4":   # add_col(bias).silu().clamp(-6, 6)
        bias = orc.f32_to_bf16_bits((rng.standard_normal(n) * 0.1).astype(np.float32)) if bf16 else \
            orc.f32_to_f16_bits((rng.standard_normal(n) * 0.1).astype(np.float32))
        epi = sg.Epilogue(dt).add_col(to_dev(bias)).silu().clamp(-6.0, 6.0)
        nodes = orc.Nodes([(4, 0, 0.0, bias, 0), (9, 0, -6.0, None, 0), (10, 0, 6.0, None, 0), (8, 3, 0.0, None, 0)])
    c = torch.full((m, n), 9.0, dtype=torch.bfloat16 if bf16 else torch.float16, device="cuda")
    fn = (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep) if epi is not None else (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)
    fn(*((to_dev(a_bits), w, c, m, epi) if epi is not None else (to_dev(a_bits), w, c, m)))
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    got = orc.t_bits_to_f32(bits_of(c), bf16)
    if sample_rows is None:
        want = orc.t_bits_to_f32(orc.matmul_q4(a_bits, q, s, None, n, k, block, m, nodes, bf16), bf16)
        return max_rel(got, want)
    wdeq = orc.q4_dequant(q, s, None, n, k, block, bf16)
    worst = 0.0
    for r0 in sample_rows:
        want = orc.matmul_q4(a_bits, q, s, None, n, k, block, m, nodes, bf16, wdeq=wdeq, first=r0, rows=1)
        worst = max(worst, max_rel(got[r0], orc.t_bits_to_f32(want[r0], bf16)))
    return worst


# tests/correctness/q4.rs:132,199-203,422 and src/kernels/lowbit/matmul.rs:534-541 shapes
@pytest.mark.parametrize("m,n,k,block", [(64, 96, 128, 32), (65, 33, 256, 32), (800, 520, 512, 32), (40, 4200, 2048, 32),
                                         (200, 4100, 2048, 32), (33, 130, 512, 16), (96, 4130, 1024, 8), (300, 200, 4096, 128),
                                         (513, 256, 576, 64)])
@pytest.mark.parametrize("bf16", [False, True])
def test_q4_gemm_matches_oracle(m, n, k, block, bf16):
    mr = run(m, n, k, block, bf16)
    assert mr <= TOL, f"{m}x{n}x{k} block {block} bf16={bf16}: max_rel {mr}"


@pytest.mark.parametrize("m,n,k,block", [(33, 4200, 2048, 64), (64, 4130, 2048, 128), (48, 4200, 2056, 256), (65, 2400, 2048, 64), (100, 2066, 2048, 128),
                                         (257, 1040, 2048, 256), (300, 520, 4096, 128), (513, 1032, 576, 64), (800, 1040, 512, 32), (512, 1040, 1000, 512)])
@pytest.mark.parametrize("bf16", [False, True])
def test_tensor_core_gemm_k_blocks(m, n, k, block, bf16):
    """K-blocks of 64 and up on the tensor-core kernel, whose stages then share scale rows: one- and two-unit stages, single
    CTAs and pairs, depth splits."""
    assert takes_gemm(m, n, k, bf16)
    mr = run(m, n, k, block, bf16)
    assert mr <= TOL, f"{m}x{n}x{k} block {block} bf16={bf16}: max_rel {mr}"


@pytest.mark.parametrize("m,n,k", [(100, 300, 512), (100, 4120, 2048), (300, 2080, 2048)])
@pytest.mark.parametrize("bf16", [False, True])
def test_q4_gemm_epilogue_graph(m, n, k, bf16):
    assert takes_gemm(m, n, k, bf16, act=True) == (n > 300)
    assert run(m, n, k, 32, bf16, ep="cfg4") <= (TOL_BF16_EP if bf16 else TOL)


def test_ragged_depth_runs_through_a_padded_copy():
    """k % 8 != 0 cannot use a tensor map: the activations are copied to rows that can, on either kernel."""
    assert run(40, 200, 1030, 32, False) <= TOL and not takes_gemm(40, 200, 1030)
    assert run(70, 2400, 2045, 32, False) <= TOL and takes_gemm(70, 2400, 2045)
    assert run(96, 130, 1027, 1, False) <= TOL


def test_config4_prefill_full_size_sampled_rows():
    """M=512, K=4096, N=14336 bf16, add_col(bias).silu().clamp(-6,6); 12 sampled rows against the oracle."""
    rows = [0, 1, 127, 128, 255, 256, 300, 383, 384, 500, 510, 511]
    mr = run(512, 14336, 4096, 32, True, seed=4, ep="cfg4", sample_rows=rows)
    assert mr <= TOL_BF16_EP, mr


def test_mlp_block_m256_sampled_rows():
    """config 5 at M=256 (hidden 4096, intermediate 14336): sampled rows against the oracle block."""
    d, f, m = 4096, 14336, 256
    rng = np.random.default_rng(55)
    wg = (rng.standard_normal((f, d)) * 0.02).astype(np.float32)
    wu = (rng.standard_normal((f, d)) * 0.02).astype(np.float32)
    wd = (rng.standard_normal((d, f)) * 0.02).astype(np.float32)
    up = sg.GatedLinear.quantize(wg, wu, sg.WeightLayout.OutIn, f, d, sg.Gate.Silu)
    down = sg.Linear.quantize(wd, sg.WeightLayout.OutIn, d, f)
    mlp = sg.Mlp.gated(up, down)
    x = torch.from_numpy(rng.standard_normal((m, d)).astype(np.float16)).cuda()
    y = torch.zeros((m, d), dtype=torch.float32, device="cuda")
    mlp.accumulate(x, y, m)
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    both_w = sg.interleave_gate_up(wg, wu, sg.WeightLayout.OutIn, f, d)
    guq, gus, _ = orc.q4_quantize(both_w, 1, 2 * f, d)
    dq, ds, _ = orc.q4_quantize(wd, 0, d, f)
    orc.set_threads(orc.max_threads())
    xs = x.cpu().numpy()
    got = y.cpu().numpy()
    for r0 in (0, 100, 255):
        want = np.zeros((1, d), np.float32)
        orc.mlp_accumulate(xs[r0:r0 + 1], want, 1, d, f, guq, gus, dq, ds)
        assert max_rel(got[r0], want[0]) <= TOL
    orc.set_threads(1)


def _big_q4(rng, n, k):
    """Random 4-bit weights too large for the warp-level kernels' share of rows, and their values in f32 on the device."""
    nbk = -(-k // 32)
    quants = rng.integers(0, 256, (k * n + 1) // 2).astype(np.uint8)
    scales = (rng.uniform(0.5, 1.5, (n, nbk)) * 0.01).astype(np.float16)
    w = sg.Q4Weights.new(quants, scales.view(np.uint16).reshape(-1), n, k)
    q = torch.from_numpy(quants).cuda()
    codes = torch.stack((q & 15, q >> 4), 1).reshape(-1)[:k * n].view(k, n).float()
    codes = torch.where(codes >= 8, codes - 16, codes)
    return w, codes * torch.from_numpy(scales.astype(np.float32)).cuda().t().repeat_interleave(32, 0)[:k]


@pytest.mark.parametrize("n,k", [(9301, 4104), (4096, 14336)])
def test_tensor_core_gemm_on_large_matrices(n, k):
    """Every form of the stage (two units, one unit, pairs of CTAs, one and two accumulator sets and token halves) and of the
    depth-split reduce, with rows, columns and depths missing: product, bias + gelu, partial sums, accumulated sums."""
    rng = np.random.default_rng(n)
    w, dense = _big_q4(rng, n, k)
    for bf16 in (False, True):
        assert takes_gemm(33, n, k, bf16)
        dt = torch.bfloat16 if bf16 else torch.float16
        rounded = dense.to(dt).float()
        bias = torch.randn(n, device="cuda").mul(0.1).to(dt)
        for m in (33, 64, 65, 100, 130, 257, 512):
            a = torch.randn(m, k, device="cuda").to(dt)
            want = a.float() @ rounded
            scale = want.abs().mean()
            c = torch.full((m, n), 9.0, dtype=dt, device="cuda")
            (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)(a, w, c, m)
            # one rounding of the store (2^-11, 2^-8 of the value) and f32 sums in another order
            assert ((c.float() - want).abs() <= (2.0 ** -8 if bf16 else 2.0 ** -11) * want.abs() + 1e-4 * scale).all(), (m, bf16)
            (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep)(a, w, c, m, sg.Epilogue("bf16" if bf16 else "f16").add_col(bias).gelu())
            ref = torch.nn.functional.gelu(want.to(dt).float() + bias.float(), approximate="tanh")
            assert ((c.float() - ref).abs() <= (2.0 ** -6 if bf16 else 2.0 ** -9) * (1 + ref.abs()) * max(1.0, float(scale))).all(), (m, bf16)
            if bf16:
                continue
            part = torch.full((m, n), 9.0, device="cuda")
            sg.Linear.from_q4(w).partial(a, part, m)
            assert (part - want).abs().max() <= 1e-4 * max(1.0, float(want.abs().max()))
            y = torch.ones((m, n), device="cuda")
            sg.Linear.from_q4(w).accumulate(a, y, m)
            sg.matmul_q4(a, w, c, m)
            assert torch.equal(y, 1 + c.float()), m
    assert sg.last_status() == 0


@pytest.mark.parametrize("m", [17, 64, 90, 200, 300])
def test_gated_block_on_large_matrices(m):
    """Gate and up columns in the two accumulator sets of every token tile, the residual add behind a depth split."""
    rng = np.random.default_rng(m)
    d, f = 4096, 9408
    assert takes_gemm(m, 2 * f, d) and takes_gemm(m, d, f)
    up, wu = _big_q4(rng, 2 * f, d)
    down, wd = _big_q4(rng, d, f)
    x = torch.randn(m, d, device="cuda").half()
    y = torch.randn(m, d, device="cuda")
    both = (x.float() @ wu.half().float()).half().float().view(m, f // 32, 2, 32)
    hid = (torch.nn.functional.silu(both[:, :, 0]) * both[:, :, 1]).reshape(m, f).half()
    out = (hid.float() @ wd.half().float()).half().float()
    got = y.clone()
    sg.Mlp.gated(sg.GatedLinear(sg.Linear.from_q4(up), sg.Gate.Silu), sg.Linear.from_q4(down)).accumulate(x, got, m)
    torch.cuda.synchronize()
    # f16 roundings of hidden units flip by one place between the orders of summation: 2^-11 each, averaged over the depth
    err, ref = (got - y - out).double(), out.double()
    assert float(err.norm() / ref.norm()) <= 1e-3 and sg.last_status() == 0
