"""Q4 GEMV / small-M GEMM on the GPU against the CPU oracle (the restated
portable path of the reference), through the C ABI.

Tolerances (float outputs): against the oracle, which also accumulates in f32
over the same weights, max |g-w|/(1+|w|) <= 1e-2 flat; against an f64 product of
the same dequantised weights, the reference's sqrt(k)-scaled bound
max(1e-2, 1e-2*sqrt(k)/4) (tests/correctness/q4.rs:56 uses 3e-2 for its
f16-accumulating kernels)."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as orc
import sme_gemm_b200 as sg
from gpu_util import bf16_bits_dev, bits_of, f16_bits_dev, half_tol, max_rel, q4_logical, takes_gemm
from refgen import Lcg

pytestmark = pytest.mark.gpu
TOL = 1e-2

# tests/correctness/gemv.rs:234-243
GEMV_SHAPES = [(1, 33, 256), (1, 389, 1027), (1, 1100, 2051), (2, 100, 70), (3, 129, 1027), (4, 4109, 4099),
               (5, 70, 513), (7, 1030, 2050)]


def run_q4(m, n, k, block, bf16=False, ep_builder=None, seed=0, from_f32=True, host=False):
    rng = np.random.default_rng(seed + m * 131 + n * 17 + k)
    q, s = q4_logical(rng, n, k, block, from_f32)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(block))
    a32 = rng.standard_normal((m, k)).astype(np.float32)
    a_bits = orc.f32_to_bf16_bits(a32) if bf16 else orc.f32_to_f16_bits(a32)
    nodes, ep = None, None
    if ep_builder is not None:
        ep_np, ep_dev, items = ep_builder(rng, m, n, bf16)
        ep = ep_np if host else ep_dev
        nodes = orc.Nodes(items)
    want = orc.matmul_q4(a_bits, q, s, None, n, k, block, m, nodes, bf16)
    if host:
        c = np.full((m, n), 0x4880, np.uint16)
        a_host = a_bits if bf16 else a_bits.view(np.float16)
        fn = (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep) if ep is not None else (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)
        fn(*((a_host, w, c, m, ep) if ep is not None else (a_host, w, c, m)))
        got = c
    else:
        a_dev = bf16_bits_dev(a_bits) if bf16 else f16_bits_dev(a_bits)
        c = torch.full((m, n), 9.0, dtype=a_dev.dtype, device="cuda")
        fn = (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep) if ep is not None else (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)
        fn(*((a_dev, w, c, m, ep) if ep is not None else (a_dev, w, c, m)))
        torch.cuda.synchronize()
        got = bits_of(c)
    assert sg.last_status() == 0
    g32, w32 = orc.t_bits_to_f32(got, bf16), orc.t_bits_to_f32(want, bf16)
    return g32, w32, (q, s, a_bits)


def q4_exact(q, s, n, k, block):
    """The weights themselves, code x scale without a rounding, [k][n] f64."""
    nib = np.stack((q & 15, q >> 4), 1).reshape(-1)[:k * n].reshape(k, n).astype(np.int64)
    scales = orc.f16_bits_to_f32(s).reshape(n, -1).astype(np.float64)
    return np.where(nib < 8, nib, nib - 16) * scales.T[np.arange(k) // block]


def bias_relu(rng, m, n, bf16):
    """add_col(bias).relu() (tests/correctness/gemv.rs Q4 epilogue case)."""
    b32 = (rng.standard_normal(n) * 0.1).astype(np.float32)
    bits = orc.f32_to_bf16_bits(b32) if bf16 else orc.f32_to_f16_bits(b32)
    dt = "bf16" if bf16 else "f16"
    ep_np = sg.Epilogue(dt).add_col(bits if bf16 else bits.view(np.float16)).relu()
    ep_dev = sg.Epilogue(dt).add_col(bf16_bits_dev(bits) if bf16 else f16_bits_dev(bits)).relu()
    return ep_np, ep_dev, [(4, 0, 0.0, bits, 0), (8, 1, 0.0, None, 0)]


@pytest.mark.parametrize("m,n,k", GEMV_SHAPES)
@pytest.mark.parametrize("block", [16, 32, 64])
def test_q4_gemv_f16_matches_oracle(m, n, k, block):
    g, w, (q, s, a_bits) = run_q4(m, n, k, block)
    mr = max_rel(g, w)
    assert mr <= TOL, f"{m}x{n}x{k} block {block}: max_rel {mr}"
    # and against an f64 product over the same dequantised weights
    wd = orc.f16_bits_to_f32(orc.q4_dequant(q, s, None, n, k, block)).astype(np.float64)
    want64 = orc.f16_bits_to_f32(a_bits).astype(np.float64).reshape(m, k) @ wd
    assert max_rel(g, want64) <= half_tol(1e-2, k)


@pytest.mark.parametrize("m,n,k", [(1, 33, 256), (3, 129, 1027), (7, 1030, 2050)])
@pytest.mark.parametrize("block", [16, 32, 64])
def test_q4_gemv_bias_relu_epilogue(m, n, k, block):
    g, w, _ = run_q4(m, n, k, block, ep_builder=bias_relu)
    assert max_rel(g, w) <= TOL


@pytest.mark.parametrize("m,n,k", [(1, 33, 256), (2, 100, 70), (5, 70, 513), (4, 1030, 1027)])
@pytest.mark.parametrize("block", [16, 32, 128])
def test_q4_gemv_bf16_matches_oracle(m, n, k, block):
    g, w, _ = run_q4(m, n, k, block, bf16=True)
    assert max_rel(g, w) <= TOL
    g, w, _ = run_q4(m, n, k, block, bf16=True, ep_builder=bias_relu)
    assert max_rel(g, w) <= TOL


@pytest.mark.parametrize("block", [1, 2, 8])
def test_q4_tiny_blocks(block):
    """tests/correctness/q4.rs:199-203 runs blocks 1 and 2."""
    g, w, _ = run_q4(3, 70, 130, block, from_f32=False)
    assert max_rel(g, w) <= TOL


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 12, 17, 33, 64])
def test_q4_row_counts_either_side_of_the_row_group(m):
    """tests/correctness/model.rs:19-76 checks m in {1,3,7,8,9,64} across the kernel switch."""
    g, w, _ = run_q4(m, 160, 320, 32)
    assert max_rel(g, w) <= TOL


def test_q4_random_byte_codes_reference_generator():
    """q4_resident (tests/correctness/q4.rs:60-123): random code bytes, scales 0.01 + 0.001*(i%5)."""
    for (m, n, k) in [(1, 1, 1), (7, 5, 3), (31, 31, 31), (32, 32, 32), (33, 17, 9), (64, 96, 48), (7, 50, 200)]:
        s = Lcg(0x44449999dead0001 ^ (m * 131 + n * 17 + k))
        a = s.fill(m * k)
        nbk = -(-k // 32)
        quants = s.bytes((k * n + 1) // 2)
        scales = orc.f32_to_f16_bits((0.01 + 0.001 * (np.arange(n * nbk) % 5)).astype(np.float32))
        w = sg.Q4Weights.new(quants, scales, n, k)
        c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
        sg.matmul_q4(torch.from_numpy(a).cuda(), w, c, m)
        want = orc.matmul_q4(a, quants, scales, None, n, k, 32, m)
        assert max_rel(c.float().cpu().numpy(), orc.f16_bits_to_f32(want)) <= TOL


def test_empty_graph_equals_plain_call_bit_for_bit():
    """tests/correctness/q4.rs:509-513."""
    m, n, k = 3, 129, 1027
    rng = np.random.default_rng(3)
    q, s = q4_logical(rng, n, k, 32)
    w = sg.Q4Weights.new(q, s, n, k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16)).cuda()
    c1 = torch.zeros((m, n), dtype=torch.float16, device="cuda")
    c2 = torch.zeros_like(c1)
    sg.matmul_q4(a, w, c1, m)
    sg.matmul_q4_ep(a, w, c2, m, sg.Epilogue())
    assert torch.equal(c1.view(torch.int16), c2.view(torch.int16))


@pytest.fixture
def stream_every_size(monkeypatch):
    """The streaming decode kernel normally takes only matrices of a few hundred KB per SM; the tuning
    knob (read per call by the library) sends every call that fits it there."""
    monkeypatch.setenv("SMEG_Q4_STREAM", "2")


# k % 8 == 0 (rows of A travel by bulk copy); n and k chosen so that column groups are cut by the
# per-CTA ranges, stages end short, and the last column group is partly outside the matrix
STREAM_SHAPES = [(1, 33, 256), (1, 4109, 4096), (3, 1030, 2056), (4, 100, 72), (7, 2000, 1032), (8, 160, 11008),
                 (9, 389, 1024), (16, 1100, 2048), (2, 16, 14336)]


@pytest.mark.parametrize("m,n,k", STREAM_SHAPES)
@pytest.mark.parametrize("block", [16, 32, 128])
def test_q4_streaming_decode_kernel_matches_oracle(stream_every_size, m, n, k, block):
    g, w, _ = run_q4(m, n, k, block)
    assert max_rel(g, w) <= TOL, f"{m}x{n}x{k} block {block}"
    g, w, _ = run_q4(m, n, k, block, ep_builder=bias_relu)
    assert max_rel(g, w) <= TOL
    if block != 16:
        g, w, _ = run_q4(m, n, k, block, bf16=True)
        assert max_rel(g, w) <= TOL


@pytest.mark.parametrize("block", [8, 4096])
def test_q4_streaming_decode_kernel_block_extremes(stream_every_size, block):
    g, w, _ = run_q4(3, 200, 8192 if block == 4096 else 264, block, from_f32=False)
    assert max_rel(g, w) <= TOL


def test_q4_streaming_decode_kernel_is_repeatable_and_leaves_its_counters_clear(stream_every_size):
    """Column groups cut between CTAs are summed in range order by whichever CTA arrives last: the result
    does not depend on which one that is, and the arrival counters are zero again for the next call."""
    m, n, k = 2, 1200, 4096
    rng = np.random.default_rng(11)
    q, s = q4_logical(rng, n, k, 32)
    w = sg.Q4Weights.new(q, s, n, k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16)).cuda()
    outs = []
    for _ in range(5):
        c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
        sg.matmul_q4(a, w, c, m)
        outs.append(c)
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    for c in outs[1:]:
        assert torch.equal(c.view(torch.int16), outs[0].view(torch.int16))


def test_q4_streaming_decode_kernel_at_the_size_that_selects_it():
    """Down projection of the MLP block at two rows: large enough to stream without the knob."""
    g, w, _ = run_q4(2, 4096, 14336, 32, seed=2)
    assert max_rel(g, w) <= TOL


def test_config1_decode_gemv_full_size():
    """M=1, K=4096, N=4096, A ~ N(0,1) f16, W ~ N(0,0.02) -> Q4_0 block 32."""
    g, w, _ = run_q4(1, 4096, 4096, 32, seed=1)
    mr = max_rel(g, w)
    assert mr <= TOL, mr


def test_host_pointer_entry_and_pack_roundtrip_through_the_device():
    g, w, (q, s, _) = run_q4(2, 100, 70, 32, host=True)
    assert max_rel(g, w) <= TOL
    g, w, _ = run_q4(3, 129, 1027, 32, host=True, ep_builder=bias_relu)
    assert max_rel(g, w) <= TOL
    wt = sg.Q4Weights.new(q, s, 100, 70)
    q2, s2 = wt.unpack()
    assert np.array_equal(q2, q) and np.array_equal(s2, s)


def test_drop_in_entry_takes_the_reference_band_major_arrays():
    """gemm_sme_f16f16_q4 / gemm_sme_b16b16_q4 with the arrays a reference-side
    Q4Weights holds (src/kernels/q4/weights.rs:92-113)."""
    m, n, k, block = 3, 200, 300, 32
    rng = np.random.default_rng(5)
    q, s = q4_logical(rng, n, k, block)
    nib, sc, _ = orc.q4_pack_band(q, s, None, n, k, block)
    a32 = rng.standard_normal((m, k)).astype(np.float32)
    L = sg.lib()
    for bf16 in (False, True):
        a_bits = orc.f32_to_bf16_bits(a32) if bf16 else orc.f32_to_f16_bits(a32)
        c = np.zeros((m, n), np.uint16)
        if bf16:
            rc = L.gemm_sme_b16b16_q4(m, n, k, c.ctypes.data, a_bits.ctypes.data, nib.ctypes.data, sc.ctypes.data, None,
                                      None, None, block, None)
        else:
            rc = L.gemm_sme_f16f16_q4(m, n, k, c.ctypes.data, a_bits.ctypes.data, nib.ctypes.data, sc.ctypes.data, None,
                                      block, None)
        assert rc == 0
        want = orc.matmul_q4(a_bits, q, s, None, n, k, block, m, None, bf16)
        assert max_rel(orc.t_bits_to_f32(c, bf16), orc.t_bits_to_f32(want, bf16)) <= TOL
    L.smeg_forget(nib.ctypes.data)
    # rc contract: bad block size -> -1 and dst untouched (csrc/gemm_f16f16_q4.h:474)
    c = np.full((m, n), 7, np.uint16)
    assert L.gemm_sme_f16f16_q4(m, n, k, c.ctypes.data, a_bits.ctypes.data, nib.ctypes.data, sc.ctypes.data, None, 24, None) == -1
    assert (c == 7).all()


def test_length_contracts_raise_like_the_reference_panics():
    q, s = q4_logical(np.random.default_rng(0), 16, 32, 32)
    w = sg.Q4Weights.new(q, s, 16, 32)
    a = torch.zeros(31, dtype=torch.float16, device="cuda")
    c = torch.zeros(16, dtype=torch.float16, device="cuda")
    with pytest.raises(AssertionError, match="a is m\\*k"):
        sg.matmul_q4(a, w, c, 1)
    with pytest.raises(AssertionError, match="col operand"):
        sg.matmul_q4_ep(torch.zeros(32, dtype=torch.float16, device="cuda"), w, c, 1,
                        sg.Epilogue().add_col(torch.zeros(15, dtype=torch.float16, device="cuda")))
    # m == 0: nothing touched
    sg.matmul_q4(torch.zeros(0, dtype=torch.float16, device="cuda"), w, torch.zeros(0, dtype=torch.float16, device="cuda"), 0)


# ---- Q4_1: the affine form (weight = scale * code + min) ----

@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("m,n,k,block", [(1, 33, 256, 32), (3, 129, 1027, 32), (7, 200, 513, 64), (64, 300, 1024, 32), (130, 257, 2050, 128)])
def test_affine_weights_match_the_scalar_statement(m, n, k, block, bf16):
    """tests/correctness/q4.rs:272-328 on the GPU: quantised with per-block minima, the product runs on the weights
    round_T(f64(scale) * code + f64(min)) (dequant_rows, src/kernels/q4/weights.rs:250-256) with f32 accumulation."""
    rng = np.random.default_rng(900 + m + n + k)
    w32 = (rng.standard_normal((n, k)) * 0.05 + 0.02).astype(np.float32)
    q, s, mins = orc.q4_quantize(w32, 0, n, k, block, True)
    w = sg.Q4Weights.with_params(q, s, mins, n, k, sg.Q4Params(block).affine())
    a32 = rng.standard_normal((m, k)).astype(np.float32)
    a_bits = orc.f32_to_bf16_bits(a32) if bf16 else orc.f32_to_f16_bits(a32)
    bias = (rng.standard_normal(n) * 0.1).astype(np.float32)
    b_bits = orc.f32_to_bf16_bits(bias) if bf16 else orc.f32_to_f16_bits(bias)
    b_dev = bf16_bits_dev(b_bits) if bf16 else f16_bits_dev(b_bits)
    ep = sg.Epilogue("bf16" if bf16 else "f16").add_col(b_dev).relu()
    want = orc.matmul_q4(a_bits, q, s, mins, n, k, block, m, orc.Nodes([(4, 0, 0.0, b_bits, 0), (8, 1, 0.0, None, 0)]), bf16)
    a_dev = bf16_bits_dev(a_bits) if bf16 else f16_bits_dev(a_bits)
    c = torch.full((m, n), 9.0, dtype=a_dev.dtype, device="cuda")
    (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep)(a_dev, w, c, m, ep)
    torch.cuda.synchronize()
    assert sg.last_status() == 0
    g32, w32o = orc.t_bits_to_f32(bits_of(c), bf16), orc.t_bits_to_f32(want, bf16)
    assert max_rel(g32, w32o) <= (2e-2 if bf16 else TOL)


def test_affine_with_zero_minima_equals_the_scale_form_and_the_library_quantiser_agrees():
    """Scale == Affine(zero mins) (tests/correctness/q4.rs:300-328), and Q4Weights.quantize with the affine parameter
    produces the oracle's codes, scales and minima."""
    rng = np.random.default_rng(77)
    m, n, k, block = 5, 96, 512, 32
    q, s = q4_logical(rng, n, k, block)
    a = f16_bits_dev(orc.f32_to_f16_bits(rng.standard_normal((m, k)).astype(np.float32)))
    scale_form = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(block))
    affine = sg.Q4Weights.with_params(q, s, np.zeros(n * (k // block), np.uint16), n, k, sg.Q4Params(block).affine())
    c0 = torch.zeros((m, n), dtype=torch.float16, device="cuda")
    c1 = torch.zeros_like(c0)
    sg.matmul_q4(a, scale_form, c0, m)
    sg.matmul_q4(a, affine, c1, m)
    assert max_rel(c1.float().cpu().numpy(), c0.float().cpu().numpy()) <= 3e-3      # f16 block sums against f32 accumulation
    w32 = (rng.standard_normal((n, k)) * 0.05 + 0.01).astype(np.float32)
    wq = sg.Q4Weights.quantize(w32, sg.WeightLayout.OutIn, n, k, sg.Q4Params(block).affine())
    qo, so, mo = orc.q4_quantize(w32, 0, n, k, block, True)
    want = orc.matmul_q4(bits_of(a), qo, so, mo, n, k, block, m)
    sg.matmul_q4(a, wq, c1, m)
    assert max_rel(c1.float().cpu().numpy(), orc.f16_bits_to_f32(want).reshape(m, n)) <= TOL


@pytest.mark.parametrize("m,n,k,off", [(1, 33, 9, 0), (4, 130, 1027, 0), (2, 70, 96, 1), (3, 40, 515, 0), (9, 65, 1501, 0), (16, 130, 64, 1),
                                       (17, 2051, 1500, 0), (65, 129, 1027, 0), (130, 300, 513, 0), (300, 140, 2049, 0)])
@pytest.mark.parametrize("bf16", [False, True])
def test_rows_off_the_16_byte_grid(m, n, k, off, bf16):
    """Depths that are no multiple of 8 and matrices that start off a 16-byte boundary, on every kernel: what lies around A
    (and between the rows' ends and the next 16-byte boundary) is non-finite and must not be read into the sums."""
    rng = np.random.default_rng(m + n + k)
    q, s = q4_logical(rng, n, k, 32)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(32))
    a32 = rng.standard_normal((m, k)).astype(np.float32)
    a_bits = (orc.f32_to_bf16_bits if bf16 else orc.f32_to_f16_bits)(a32)
    room = torch.full((m * k + 64,), float("nan"), dtype=torch.bfloat16 if bf16 else torch.float16, device="cuda")
    a = room[off:off + m * k]
    a.copy_((bf16_bits_dev if bf16 else f16_bits_dev)(a_bits).reshape(-1))
    c = torch.full((m, n), 9.0, dtype=a.dtype, device="cuda")
    (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)(a, w, c, m)
    torch.cuda.synchronize()
    want = orc.matmul_q4(a_bits, q, s, None, n, k, 32, m, None, bf16)
    assert sg.last_status() == 0
    assert max_rel(orc.t_bits_to_f32(bits_of(c), bf16), orc.t_bits_to_f32(want, bf16)) <= TOL


@pytest.mark.parametrize("m,n,k,block", [(1, 16, 64, 32), (3, 17, 72, 32), (8, 33, 520, 64), (5, 4800, 128, 32), (9, 1152, 1536, 128), (16, 9500, 264, 32),
                                         (13, 100, 8200, 256), (17, 65, 4096, 32), (33, 640, 1000, 32), (64, 1152, 1536, 64)])
@pytest.mark.parametrize("bf16", [False, True])
def test_warp_level_kernel(m, n, k, block, bf16):
    """Row tiles of 8 and 16 with rows missing, passes of one and two column groups with a group missing, depths that leave
    warps without a unit or end inside one, an epilogue on the product."""
    got, want, (q, s, a_bits) = run_q4(m, n, k, block, bf16, bias_relu, from_f32=False)
    assert max_rel(got, want) <= (2e-2 if bf16 else TOL)       # one bf16 place of the product can flip through the epilogue
    # the product itself: f32 sums (2^-24 of the terms' sizes a few times over) of the weights code x scale, unrounded, and one
    # rounding of the store -- for bf16 as for f16, whatever the rows of the call
    got, want, (q, s, a_bits) = run_q4(m, n, k, block, bf16, None)
    assert max_rel(got, want) <= TOL
    if bf16 or m > 2:                                          # (one and two f16 rows run on the one-wave kernel)
        a64, wt = orc.t_bits_to_f32(a_bits, bf16).reshape(m, k).astype(np.float64), q4_exact(q, s, n, k, block)
        exact, room = a64 @ wt, np.abs(a64) @ np.abs(wt)
        assert (np.abs(got.reshape(m, n) - exact) <= 2.0 ** (-8 if bf16 else -11) * np.abs(exact) + 2.0 ** -25 + 2.0 ** -21 * room).all()


@pytest.mark.parametrize("m", [1, 2, 3, 8, 16, 17, 40, 64])
@pytest.mark.parametrize("d,f", [(256, 640), (1024, 3072), (252, 672)])
def test_gated_block_in_two_launches_is_its_separate_passes(m, d, f):
    """The gated product and the residual add in the stores of the products, at every row count that fuses them, on whole and
    on ragged rows: the bits of product, gate pass, product, add."""
    rng = np.random.default_rng(m + d)
    w = [(rng.standard_normal((f, d)) * 0.05).astype(np.float32) for _ in range(2)]
    up = sg.GatedLinear.quantize(w[0], w[1], sg.WeightLayout.OutIn, f, d, sg.Gate.Silu)
    down = sg.Linear.quantize((rng.standard_normal((d, f)) * 0.05).astype(np.float32), sg.WeightLayout.OutIn, d, f)
    x = torch.from_numpy(rng.standard_normal((m, d)).astype(np.float16)).cuda()
    y = torch.from_numpy(rng.standard_normal((m, d)).astype(np.float32)).cuda()
    want = y.clone()
    sg.Mlp.gated(up, down).accumulate(x, y, m)
    hid = torch.empty((m, f), dtype=torch.float16, device="cuda")
    up.forward(x, hid, m)
    out = torch.empty((m, d), dtype=torch.float16, device="cuda")
    down.forward(hid, out, m)
    want += out.float()
    torch.cuda.synchronize()
    assert sg.last_status() == 0 and torch.equal(y, want)


@pytest.mark.parametrize("magnitude", [1e4, 1.0, 1e-4])
@pytest.mark.parametrize("m,n,k,off", [(1, 130, 1027, 0), (1, 70, 96, 1), (2, 130, 1500, 0), (2, 2051, 1027, 1), (3, 130, 1500, 0),
                                       (1, 9600, 66, 0), (2, 9700, 523, 0), (2, 9600, 258, 1), (2, 64, 8190, 0), (2, 40, 20001, 0)])
def test_rows_off_the_16_byte_grid_keep_f32_sums(m, n, k, off, magnitude):
    """Activations whose products leave f16's range on both sides: the product is the exact one to its store's rounding.  Rows
    that start on every boundary, passes of one and two column groups, depths whose rows are staged and too long for it."""
    rng = np.random.default_rng(m + n + k)
    q, s = q4_logical(rng, n, k, 32)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(32))
    a16 = (rng.standard_normal((m, k)) * magnitude).astype(np.float16)
    room = torch.full((m * k + 64,), float("nan"), dtype=torch.float16, device="cuda")
    a = room[off:off + m * k]
    a.copy_(torch.from_numpy(a16.reshape(-1)).cuda())
    c = torch.full((m, n), 9.0, dtype=torch.float16, device="cuda")
    sg.matmul_q4(a, w, c, m)
    torch.cuda.synchronize()
    wt, a64 = q4_exact(q, s, n, k, 32), a16.astype(np.float64)
    want, room = a64 @ wt, np.abs(a64) @ np.abs(wt)
    # half a place of the f16 store (2^-25 on its subnormal grid), and f32 sums in any order: 2^-24 of the terms' sizes a few times over
    assert (np.abs(c.cpu().numpy().astype(np.float64) - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -25 + 2.0 ** -21 * room).all()
    assert sg.last_status() == 0


@pytest.mark.parametrize("m,block,k,off", [(64, 32, 4092, 0), (40, 32, 4096, 1), (8, 16, 4092, 0), (1, 16, 4091, 0), (40, 16, 4092, 0)])
def test_rows_off_the_16_byte_grid_in_a_capture_without_a_warm_call(m, block, k, off):
    """These calls need no workspace, so the first one on a stream may be inside a capture; the replay gives the bits the
    captured kernels give, within the bar of the same call outside."""
    n = 4096
    rng = np.random.default_rng(m + k)
    q, s = q4_logical(rng, n, k, block, from_f32=False)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(block))
    a = torch.full((m * k + 64,), float("nan"), dtype=torch.float16, device="cuda")[off:off + m * k]
    a.copy_(torch.from_numpy(rng.standard_normal(m * k).astype(np.float16)).cuda())
    c, want = (torch.full((m, n), 9.0, dtype=torch.float16, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        sg.matmul_q4(a, w, c, m)
    graph.replay()
    torch.cuda.synchronize()
    sg.matmul_q4(a, w, want, m)
    torch.cuda.synchronize()
    assert max_rel(c.float().cpu().numpy(), want.float().cpu().numpy()) <= TOL and sg.last_status() == 0
    a64, wt = a.cpu().numpy().astype(np.float64).reshape(m, k), q4_exact(q, s, n, k, block)
    assert max_rel(c.float().cpu().numpy(), a64 @ wt) <= half_tol(1e-2, k)
    del graph


@pytest.mark.parametrize("form", ["f16", "bf16", "bias", "accumulate", "gated"])
def test_tensor_core_calls_in_a_capture_without_a_warm_call(form):
    """Rows and matrices on which the tensor-core GEMM splits the depth: the first such call on a stream may be inside a
    capture, where its workspace cannot be allocated, and runs on the kernel for few rows there."""
    m, n, k, block = 40, 4096, 4096, 32
    rng = np.random.default_rng(51)
    q, s = q4_logical(rng, n, k, block, from_f32=False)
    w = sg.Q4Weights.with_params(q, s, None, n, k, sg.Q4Params(block))
    assert takes_gemm(m, n, k, form == "bf16")
    dtype = torch.bfloat16 if form == "bf16" else torch.float16
    a = torch.from_numpy((rng.standard_normal((m, k)) * 0.1).astype(np.float32)).cuda().to(dtype)
    ep = sg.Epilogue("f16").add_col(torch.from_numpy(rng.standard_normal(n).astype(np.float16)).cuda())
    if form == "gated":
        wg, wu, wd = ((rng.standard_normal(n // 2 * k) * 0.02).astype(np.float32) for _ in range(3))
        mlp = sg.Mlp.gated(sg.GatedLinear.quantize(wg, wu, sg.WeightLayout.OutIn, n // 2, k, sg.Gate.Silu),
                           sg.Linear.quantize(wd, sg.WeightLayout.OutIn, n, n // 2))

    def call(c):
        if form == "f16":
            sg.matmul_q4(a, w, c, m)
        elif form == "bf16":
            sg.matmul_q4_bf16(a, w, c, m)
        elif form == "bias":
            sg.matmul_q4_ep(a, w, c, m, ep)
        elif form == "accumulate":
            sg.Linear.from_q4(w).accumulate(a, c, m)
        else:
            mlp.accumulate(a, c, m)

    f32 = form in ("accumulate", "gated")
    got, want = (torch.ones((m, n), dtype=torch.float32 if f32 else dtype, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream(priority=-1)):
        call(got)
    graph.replay()
    torch.cuda.synchronize()
    call(want)
    torch.cuda.synchronize()
    assert max_rel(got.float().cpu().numpy(), want.float().cpu().numpy()) <= TOL and sg.last_status() == 0
    del graph


# One and two rows on the kernel that takes stages of four units: depths from its first (29 units, a last stage of one unit) up,
# depths that end in a stage's middle, K-blocks of a half unit up to longer than the depth, several column groups a CTA.
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k,block", [(33, 1800, 32), (389, 2056, 64), (16, 2304, 128), (7001, 1856, 32), (100, 11008, 512), (48, 4096, 8192), (20, 14400, 32)])
def test_one_and_two_rows_by_stages_of_four_units(m, n, k, block):
    """Against the product in 64 bits of the weights themselves: an f16 store (2^-11 of the value) and f32 sums, whose terms
    code x a are exact: at most 16 roundings of 2^-24 of the largest partial sum of |code + 8| |a| scale per 256 depths."""
    g, _, (q, s, a_bits) = run_q4(m, n, k, block, seed=k)
    a = orc.f16_bits_to_f32(a_bits).astype(np.float64).reshape(m, k)
    want = a @ q4_exact(q, s, n, k, block)
    big = np.abs(a) @ np.abs(orc.f16_bits_to_f32(s).reshape(n, -1).astype(np.float64).T[np.arange(k) // block]) * 16
    assert np.all(np.abs(g - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -24 + 16 * 2.0 ** -24 * big)


@pytest.mark.parametrize("m", [1, 2])
def test_rows_with_infinities_by_stages_of_four_units(m):
    """An infinity meets a code of zero as a NaN and any other as an infinity, and leaves other rows alone."""
    n, k = 200, 2048
    rng = np.random.default_rng(4)
    q, s = q4_logical(rng, n, k, 32, from_f32=False)
    w = sg.Q4Weights.new(q, s, n, k)
    a = rng.standard_normal((m, k)).astype(np.float16)
    a[0, 1234] = np.inf
    c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
    sg.matmul_q4(torch.from_numpy(a).cuda(), w, c, m)
    exact = q4_exact(q, s, n, k, 32)
    with np.errstate(invalid="ignore"):
        want = a.astype(np.float64) @ exact
    got = c.float().cpu().numpy()
    assert np.array_equal(np.isnan(got[0]), exact[1234] == 0) and np.array_equal(np.isposinf(got[0]), exact[1234] > 0)
    assert np.all(np.isfinite(got[1:])) and max_rel(got[1:], want[1:]) <= 1e-3


@pytest.mark.parametrize("other", [0, 1])
@pytest.mark.parametrize("what", [np.inf, np.nan])
def test_a_finite_row_keeps_its_bits_beside_one_with_infinities(other, what):
    """Two rows by stages of four units: the finite one's result is that of the same call with a finite neighbour, bit for bit."""
    n, k = 200, 2048
    rng = np.random.default_rng(5)
    q, s = q4_logical(rng, n, k, 32, from_f32=False)
    w = sg.Q4Weights.new(q, s, n, k)
    a = rng.standard_normal((2, k)).astype(np.float16)
    c = [torch.zeros((2, n), dtype=torch.float16, device="cuda") for _ in range(2)]
    sg.matmul_q4(torch.from_numpy(a).cuda(), w, c[0], 2)
    a[other, 77] = what
    sg.matmul_q4(torch.from_numpy(a).cuda(), w, c[1], 2)
    assert not torch.isfinite(c[1][other]).all()
    assert torch.equal(c[0][1 - other].view(torch.int16), c[1][1 - other].view(torch.int16))


# As many CTAs an SM as have room: three become two (one and two rows), two become one.
@pytest.mark.parametrize("m,n,k,glu", [(2, 4752, 4096, False), (1, 4752, 9216, False), (2, 2400, 11008, False), (1, 2384, 24000, False), (2, 1024, 14336, False),
                                       (2, 33, 14400, False), (2, 4800, 4096, True), (2, 4800, 11008, True)])
def test_one_and_two_rows_where_fewer_ctas_fit(m, n, k, glu):
    """Against the same rows one at a time in f32 sums of the weights themselves (an f16 store, 2^-11, and f32 sums as above)."""
    rng = np.random.default_rng(n + k)
    q = rng.integers(0, 256, n * k // 2, dtype=np.uint8)
    s = rng.uniform(0.002, 0.01, n * (k // 32)).astype(np.float16)
    w = sg.Q4Weights.new(q, s.view(np.uint16), n, k)
    a = rng.standard_normal((m, k)).astype(np.float16)
    codes = torch.from_numpy(np.stack([q & 15, q >> 4], 1).astype(np.int8).reshape(k, n)).cuda()
    codes = (codes - 16 * (codes > 7)).float()
    scale = torch.from_numpy(s.astype(np.float32)).cuda().view(n, k // 32).t()
    blocks = torch.einsum("mbd,bdn->mbn", torch.from_numpy(a).cuda().double().view(m, k // 32, 32), codes.view(k // 32, 32, n).double())
    want = (blocks * scale.double()).sum(1)
    if not glu:
        c = torch.zeros((m, n), dtype=torch.float16, device="cuda")
        sg.matmul_q4(torch.from_numpy(a).cuda(), w, c, m)
        big = torch.from_numpy(np.abs(a)).cuda().double() @ (16 * scale.double().repeat_interleave(32, 0))
        assert torch.all((c.double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -24 + 16 * 2.0 ** -24 * big)
        return
    # gate and up columns interleaved by 32: the block's hidden units, rounded as the separate passes round them
    down = sg.Linear.from_q4(sg.Q4Weights.new(*q4_logical(rng, 64, n // 2, 32, from_f32=False), 64, n // 2))
    mlp = sg.Mlp.gated(sg.GatedLinear(sg.Linear.from_q4(w), sg.Gate.Silu), down)
    y = torch.zeros((m, 64), device="cuda")
    mlp.accumulate(torch.from_numpy(a).cuda(), y, m)
    v = want.view(m, n // 64, 2, 32).half().double()
    hidden = (v[:, :, 0] * torch.sigmoid(v[:, :, 0]) * v[:, :, 1]).reshape(m, n // 2).half()
    got = torch.zeros((m, 64), dtype=torch.float16, device="cuda")
    sg.matmul_q4(hidden, down.q4, got, m)
    assert max_rel(y.cpu().numpy(), got.float().cpu().numpy()) <= TOL
