"""GPU parity: MixedQLinear.forward (fused, unfused, shared input, small-M, bf16) vs the CPU oracle."""
import copy
import weakref

import pytest
import torch

from oracle import kernel_path as kp
from quik_b200 import _lib, matmul
from quik_b200.qlinear import MixedQLinear, SharedQuantizedInput
from quik_b200.workloads import make_layer
from tests.gpu_util import assert_device_clean, dev, rel_rms_err

pytestmark = pytest.mark.gpu

# BASELINE tolerance: max-abs error of the fp16 output relative to the output RMS
TOL_RMS = 1e-2


def _oracle_out(case, round_y):
    m = case.module
    buf = {"int_weight": m.int_weight.cpu(), "weights_scales": m.weights_scales.cpu(), "reduced_w": m.reduced_w.cpu(),
           "int_indices": m.int_indices.cpu(), "fp_indices": m.fp_indices.cpu(),
           "bias": None if m.bias is None else m.bias.cpu()}
    if m.fp_features_num > 0:
        buf["fp_weight"] = m.fp_weight.cpu()
    return kp.mixed_linear_forward(case.x.cpu(), buf, m.bits, round_y=round_y)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,F,bits", [
    (1, 4096, 512, 256, 4), (16, 4096, 264, 256, 4), (16, 1024, 128, 0, 8), (7, 11008, 256, 256, 8),
    (17, 4096, 512, 256, 4), (129, 4096, 520, 256, 4), (256, 1024, 384, 0, 4), (128, 11008, 256, 256, 8),
    (2048, 4096, 1024, 256, 4), (300, 8192, 1024, 1024, 4), (64, 96, 40, 32, 4),
    (40, 112, 24, 32, 4), (9, 112, 24, 32, 4),      # 80 integer columns: packed rows of 40 bytes, tiled GEMM at any M
])
def test_fused_forward_matches_oracle(dtype, M, K, N, F, bits):
    case = make_layer("t", M, K, N, bits, F=F, seed=M + N, device=dev(), dtype=dtype, clip=False)
    out = case.module(case.x.unsqueeze(0))
    assert out.shape == (1, M, N) and out.dtype == dtype
    ref = _oracle_out(case, round_y=False)
    err = rel_rms_err(out[0].cpu(), ref)
    # bf16 has 3 fewer mantissa bits: the final rounding and the storage-type rounding of the outlier
    # product are each worth up to 2^-8 of the value
    tol = TOL_RMS if dtype == torch.float16 else 4e-2
    assert err < tol, err
    # the reference's own unfused sequence rounds the outlier product to the storage type before the
    # dequantize step; in bf16 that extra rounding alone is worth up to 2^-8 of |y|
    ref_rounded = _oracle_out(case, round_y=True)
    assert rel_rms_err(out[0].cpu(), ref_rounded) < tol
    out2 = case.module(case.x.unsqueeze(0))
    assert torch.equal(out, out2)                            # deterministic
    assert_device_clean()


@pytest.mark.parametrize("col_pad", [8, 3])
@pytest.mark.parametrize("engine", [_lib.ENGINE_TCGEN05, _lib.ENGINE_TCGEN05_TS], ids=["smem_operands", "tmem_operand"])
@pytest.mark.parametrize("tile,pair", [(0, 0), (240, 2), (144, 2), (176, 1)])
@pytest.mark.parametrize("M,K,N,F,bits", [(300, 1088, 520, 64, 4), (129, 1088, 264, 64, 8), (257, 608, 1000, 32, 4),
                                          (16, 1088, 520, 64, 4), (100, 1088, 520, 64, 8)])
def test_fused_layer_writes_only_its_columns(M, K, N, F, bits, tile, pair, engine, col_pad):
    """The layer's output is a window of a poisoned slab (rows and columns of padding on every side, handed over as
    `out_buffer` with a row pitch wider than N): the window equals the plain forward bit for bit and the padding is
    untouched.  col_pad = 8 keeps the window 16-byte aligned (vector stores), col_pad = 3 does not (element
    stores); the tile widths end a warp's column range with a
    16-column step.  Covers the ragged-edge stores of the tiled kernel and the stores of
    the weight-streaming engines (16 and 100 tokens)."""
    case = make_layer("t", M, K, N, bits, F=F, seed=M + N, device=dev(), clip=False)
    row_pad = 5
    poison = -1234.0
    try:
        _lib.set_engine(engine)
        _lib.set_tile_n(tile)
        _lib.set_cta_pair(pair)
        want = case.module(case.x.unsqueeze(0))[0].clone()
        slab = torch.full((M + 2 * row_pad, N + 2 * col_pad), poison, dtype=torch.float16, device=dev())
        window = slab[row_pad:row_pad + M, col_pad:col_pad + N]
        case.module.out_buffer = window
        got = case.module(case.x.unsqueeze(0))[0]
        assert got.data_ptr() == window.data_ptr()
        torch.cuda.synchronize()
    finally:
        case.module.out_buffer = None
        _lib.set_engine(_lib.ENGINE_AUTO)
        _lib.set_tile_n(0)
        _lib.set_cta_pair(0)
    assert_device_clean()
    assert torch.equal(window, want)
    border = slab.clone()
    border[row_pad:row_pad + M, col_pad:col_pad + N] = poison
    assert bool((border == poison).all()), "the layer wrote outside its [M, N] window"
    assert rel_rms_err(want.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS


@pytest.mark.parametrize("F", [64, 0])
@pytest.mark.parametrize("tile,pair", [(0, 0), (48, 1), (112, 2), (256, 2)])
@pytest.mark.parametrize("N", [1, 9, 31, 250, 509])
def test_rows_that_start_anywhere_in_a_sector(N, tile, pair, F):
    """The tiled kernel's stores of rows without 16-byte alignment: windows that start at every column 0..15 of a slab whose row
    pitch moves the start on by another odd amount per row, from a single column up to parts of several sectors.  Bits equal
    those of the dense result, the rest of the slab is untouched, and so is an int32 product of N columns."""
    M, K = 131, 224 + F
    case = make_layer("t", M, K, N, 8, F=F, seed=N, device=dev(), clip=False)
    try:
        _lib.set_tile_n(tile)
        _lib.set_cta_pair(pair)
        want = case.module(case.x.unsqueeze(0))[0].clone()
        for off in range(16):
            slab = torch.full((M, N + 17 + (off & 2)), -1234.0, dtype=torch.float16, device=dev())
            case.module.out_buffer = slab[:, off:off + N]
            case.module(case.x.unsqueeze(0))
            assert torch.equal(slab[:, off:off + N], want), off
            slab[:, off:off + N] = -1234.0
            assert bool((slab == -1234.0).all()), off
        g = torch.Generator().manual_seed(N)
        a = torch.randint(-128, 128, (M, 208), generator=g, dtype=torch.int8)
        b = torch.randint(-128, 128, (N, 208), generator=g, dtype=torch.int8)
        c = matmul.int8Matmul(a.to(dev()), b.to(dev()))
        assert torch.equal(c.cpu().long(), a.long() @ b.long().t())
    finally:
        case.module.out_buffer = None
        _lib.set_tile_n(0)
        _lib.set_cta_pair(0)
    assert rel_rms_err(want.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
    assert_device_clean()


@pytest.mark.parametrize("F", [64, 0])
@pytest.mark.parametrize("tile", [32, 128, 144, 224])
@pytest.mark.parametrize("N", [3, 130, 257, 1021])
def test_rows_without_alignment_by_tile_width(N, tile, F):
    """Either side of the tile width up to which rows without 16-byte alignment are stored element by element, beyond it by sectors:
    the outputs are those of the other side, and only the layer's columns are written; an int32 product too."""
    M, K = 131, 224 + F
    case = make_layer("t", M, K, N, 8, F=F, seed=N, device=dev(), clip=False)
    g = torch.Generator().manual_seed(N)
    a = torch.randint(-128, 128, (M, 208), generator=g, dtype=torch.int8)
    b = torch.randint(-128, 128, (N, 208), generator=g, dtype=torch.int8)
    try:
        _lib.set_tile_n(80)
        want = case.module(case.x.unsqueeze(0))[0].clone()
        _lib.set_tile_n(tile)
        for pair in (1, 2):
            _lib.set_cta_pair(pair)
            for off in (0, 1, 6, 15):
                slab = torch.full((M, N + 16 + (off & 1)), -1234.0, dtype=torch.float16, device=dev())
                case.module.out_buffer = slab[:, off:off + N]
                case.module(case.x.unsqueeze(0))
                assert torch.equal(slab[:, off:off + N], want), off
                slab[:, off:off + N] = -1234.0
                assert bool((slab == -1234.0).all()), off
            c = matmul.int8Matmul(a.to(dev()), b.to(dev()))
            assert torch.equal(c.cpu().long(), a.long() @ b.long().t())
    finally:
        case.module.out_buffer = None
        _lib.set_tile_n(0)
        _lib.set_cta_pair(0)
    assert rel_rms_err(want.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
    assert_device_clean()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,F,bits", [
    (16, 256, 128, 0, 4), (16, 1280, 128, 256, 8), (1, 4352, 512, 256, 4), (16, 4352, 264, 256, 4), (7, 11264, 256, 256, 8),
    (16, 4352, 4096, 256, 4),      # K split over a cluster of 4 CTAs
    (13, 11264, 4096, 256, 8),     # ... of 8
    (16, 4352, 22016, 256, 4),     # one CTA per slab, more slabs than fit at once
    (5, 4232, 300, 72, 4),         # ragged N, K and F
])
def test_small_m_engines_agree(dtype, M, K, N, F, bits):
    """Few tokens: the three weight-streaming engines (tcgen05 with on-chip widening; mma.sync fed by direct loads or
    by a TMA ring) and the tensor-core GEMM on widened weights give the oracle's result; the integer part is exact
    in all of them."""
    case = make_layer("t", M, K, N, bits, F=F, seed=M + N, device=dev(), dtype=dtype, clip=False)
    outs = {}
    try:
        for mode in (_lib.SMALL_M_TCGEN05, _lib.SMALL_M_MMA_SYNC, _lib.SMALL_M_TMA_MMA, _lib.SMALL_M_OFF, _lib.SMALL_M_AUTO):
            _lib.set_small_m(mode)
            outs[mode] = case.module(case.x.unsqueeze(0))[0].clone()
            again = case.module(case.x.unsqueeze(0))[0]
            assert torch.equal(outs[mode], again)                # deterministic (split-K included)
    finally:
        _lib.set_small_m(_lib.SMALL_M_AUTO)
    assert_device_clean()
    ref = _oracle_out(case, round_y=False)
    tol = TOL_RMS if dtype == torch.float16 else 4e-2
    for mode, out in outs.items():
        assert rel_rms_err(out.cpu(), ref) < tol, mode
    # the engines differ only in the summation order of the outlier product: at most one unit in the last place of
    # the largest outputs (2^-10 of 4 x RMS in fp16)
    agree = 5e-3 if dtype == torch.float16 else 4e-2
    assert rel_rms_err(outs[_lib.SMALL_M_TCGEN05], outs[_lib.SMALL_M_MMA_SYNC]) < agree
    assert rel_rms_err(outs[_lib.SMALL_M_TCGEN05], outs[_lib.SMALL_M_OFF]) < agree
    assert rel_rms_err(outs[_lib.SMALL_M_TMA_MMA], outs[_lib.SMALL_M_MMA_SYNC]) < agree
    if F == 0:
        assert torch.equal(outs[_lib.SMALL_M_TCGEN05], outs[_lib.SMALL_M_MMA_SYNC])
        assert torch.equal(outs[_lib.SMALL_M_TMA_MMA], outs[_lib.SMALL_M_MMA_SYNC])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [17, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("K,N,F,bits", [(4352, 4096, 256, 4), (11264, 520, 256, 8), (1056, 300, 32, 4)])
def test_streaming_engine_up_to_128_tokens(dtype, M, K, N, F, bits):
    """17 to 128 tokens run on the tcgen05 weight-streaming engine (token operand of 64 or 128 rows, weights in
    storage format); same result as the tiled tensor-core GEMM on widened weights, and the oracle's."""
    case = make_layer("t", M, K, N, bits, F=F, seed=M + N, device=dev(), dtype=dtype, clip=False)
    try:
        out = case.module(case.x.unsqueeze(0))[0].clone()
        again = case.module(case.x.unsqueeze(0))[0]
        _lib.set_small_m(_lib.SMALL_M_OFF)
        tiled = case.module(case.x.unsqueeze(0))[0].clone()
    finally:
        _lib.set_small_m(_lib.SMALL_M_AUTO)
    assert_device_clean()
    assert torch.equal(out, again)
    tol = TOL_RMS if dtype == torch.float16 else 4e-2
    assert rel_rms_err(out.cpu(), _oracle_out(case, round_y=False)) < tol
    assert rel_rms_err(out, tiled) < (5e-3 if dtype == torch.float16 else 4e-2)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,F,bits", [(129, 1088, 520, 64, 4), (300, 4352, 1024, 256, 4), (2048, 4096, 1280, 256, 4),
                                          (257, 11264, 520, 256, 8), (513, 1024, 264, 0, 4), (400, 2080, 96, 32, 8),
                                          (1000, 4128, 4096, 32, 4)])
def test_tensor_memory_operand_engine_matches_shared_memory_engine(dtype, M, K, N, F, bits):
    """The two tcgen05 engines (token codes one per byte from shared memory; packed 4-bit codes widened on chip into
    tensor memory) compute every output element from the same exact integer sum and the same order of outlier
    products, so their results are identical bit for bit whatever tiles they pick; both match the oracle."""
    case = make_layer("t", M, K, N, bits, F=F, seed=M + N, device=dev(), dtype=dtype, clip=False)
    outs = {}
    try:
        for eng in (_lib.ENGINE_TCGEN05, _lib.ENGINE_TCGEN05_TS):
            _lib.set_engine(eng)
            outs[eng] = case.module(case.x.unsqueeze(0))[0].clone()
            assert torch.equal(outs[eng], case.module(case.x.unsqueeze(0))[0])
    finally:
        _lib.set_engine(_lib.ENGINE_AUTO)
    assert_device_clean()
    assert torch.equal(outs[_lib.ENGINE_TCGEN05], outs[_lib.ENGINE_TCGEN05_TS])
    tol = TOL_RMS if dtype == torch.float16 else 4e-2
    assert rel_rms_err(outs[_lib.ENGINE_TCGEN05_TS].cpu(), _oracle_out(case, round_y=False)) < tol


@pytest.mark.parametrize("M", [16, 300])
def test_dependent_launch_matches_stream_order(M):
    """A chain of layers (each output feeds the next quantizer) with kernels launched as programmatic dependents
    gives bit-identical results to plain stream order, eagerly and replayed from a CUDA graph."""
    cases = [make_layer(f"l{i}", M, 1024 + 64, 1024 + 64, 4 if i % 2 == 0 else 8, F=64, seed=i, device=dev(), clip=False)
             for i in range(4)]
    x0 = cases[0].x

    def chain():
        h = x0
        for c in cases:
            h = c.module(h.unsqueeze(0))[0]
            h = (h / h.float().abs().max().clamp_min(1e-3)).to(x0.dtype)     # keep magnitudes stable (a torch kernel in between)
        return h

    try:
        _lib.set_pdl(False)
        ref = chain().clone()
        _lib.set_pdl(True)
        eager = chain().clone()
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                out = chain()
            for _ in range(3):
                g.replay()
        torch.cuda.synchronize()
    finally:
        _lib.set_pdl(True)
    assert torch.equal(eager, ref)
    assert torch.equal(out, ref)
    assert_device_clean()


def test_dependent_launch_back_to_back_layers():
    """Layers launched back to back with no other kernel in between (shared quantized input: quantizer, then three
    fused launches), where a launch can overtake its predecessor's tail; outputs equal plain stream order."""
    shared = SharedQuantizedInput(3)
    cases = [make_layer(f"m{i}", 16, 4096 + 256, 1024, 4, F=256, seed=0, device=dev(), shared_input=shared, clip=False)
             for i in range(3)]
    x = cases[0].x
    res = {}
    try:
        for on in (False, True):
            _lib.set_pdl(on)
            for rep in range(3):
                res[on] = [c.module(x.unsqueeze(0)).clone() for c in cases]
        torch.cuda.synchronize()
    finally:
        _lib.set_pdl(True)
    for a, b in zip(res[False], res[True]):
        assert torch.equal(a, b)
    assert_device_clean()


@pytest.mark.parametrize("pair", [1, 2])
@pytest.mark.parametrize("M,K,N,F,bits", [(300, 4096, 520, 256, 4), (2048, 4096, 2048, 256, 4), (640, 11008, 512, 256, 8),
                                          (128, 1024, 256, 64, 4), (513, 2048, 1000, 0, 4)])
def test_fused_forward_single_cta_and_pair_agree(pair, M, K, N, F, bits):
    """Both tile schedules (one CTA per tile, CTA pair per 256-row tile) against the oracle and each other."""
    case = make_layer("t", M, K, N, bits, F=F, seed=7, device=dev(), clip=False)
    _lib.set_cta_pair(pair)
    try:
        out = case.module(case.x.unsqueeze(0))[0]
        torch.cuda.synchronize()
    finally:
        _lib.set_cta_pair(0)
    assert_device_clean()
    ref = _oracle_out(case, round_y=True)
    assert rel_rms_err(out.cpu(), ref) < TOL_RMS
    _lib.set_cta_pair(1)
    try:
        single = case.module(case.x.unsqueeze(0))[0]
    finally:
        _lib.set_cta_pair(0)
    assert rel_rms_err(out.cpu(), single.cpu()) < 2e-3      # only the outlier product's summation order differs


@pytest.mark.parametrize("M,bits,F", [(64, 4, 256), (5, 8, 0), (200, 8, 256)])
def test_unfused_forward_matches_oracle(M, bits, F):
    case = make_layer("t", M, 4096, 256, bits, F=F, seed=3, device=dev(), clip=False)
    case.module.fused = False
    out = case.module(case.x.unsqueeze(0))[0].cpu()
    ref = _oracle_out(case, round_y=True)
    # same int32 accumulators and same fp32 epilogue; only the cuBLAS outlier GEMM may round differently
    assert rel_rms_err(out, ref) < 2e-3
    case.module.fused = True
    fused = case.module(case.x.unsqueeze(0))[0].cpu()
    assert rel_rms_err(fused, out) < TOL_RMS


def test_bias_and_no_outliers():
    torch.manual_seed(0)
    K, N, M = 512, 128, 40
    lin = torch.nn.Linear(K, N, bias=True)
    w = (0.02 * torch.randn(N, K)).half()
    scales = w.float().abs().max(1, keepdim=True)[0] / 7
    mod = MixedQLinear.from_float(lin, w, scales, fp_indices=None, bits=4).to(dev())
    x = torch.randn(M, K).half().to(dev())
    out = mod(x.unsqueeze(0))[0].cpu()
    buf = kp.from_float_buffers(w, scales, None, 4, bias=lin.bias.data.half())
    ref = kp.mixed_linear_forward(x.cpu(), buf, 4, round_y=True, contract=True)
    # no outlier GEMM: exact integer GEMM + the fp32 multiply-add epilogue -> same fp16 values
    diff = (out.float() - ref.float()).abs()
    assert (diff <= ref.float().abs() * 2 ** -10 + 2.0 ** -24).all() and (diff != 0).float().mean() < 1e-4
    for name in ("int_weight", "weights_scales", "reduced_w", "int_indices", "bias"):
        assert torch.equal(getattr(mod, name).cpu(), buf[name]), name


def test_shared_quantized_input_groups():
    """q/k/v style group of three layers shares one quantizer call (experiments/llama.py:402-411)."""
    shared = SharedQuantizedInput(3)
    cases = [make_layer(f"m{i}", 48, 1024, 128, 4, F=64, seed=0, device=dev(), shared_input=shared, clip=False)
             for i in range(3)]
    x = cases[0].x
    outs = []
    for i, c in enumerate(cases):
        outs.append(c.module(x.unsqueeze(0)))
        if i < 2:
            assert shared.qint_x is not None and shared.cur_group_elem == i + 1
    assert shared.qint_x is None and shared.cur_group_elem == 0
    for c, o in zip(cases, outs):
        solo = make_layer("s", 48, 1024, 128, 4, F=64, seed=0, device=dev(), clip=False)
        assert torch.equal(o, solo.module(x.unsqueeze(0)))


def test_state_dict_round_trip():
    case = make_layer("t", 32, 1024, 128, 4, F=64, seed=1, device=dev(), clip=False)
    sd = case.module.state_dict()
    fresh = MixedQLinear(1024, 128, fp_features_num=64, bits=4)
    fresh.bias = None
    fresh.load_state_dict(sd)
    fresh = fresh.to(dev())
    assert torch.equal(fresh(case.x.unsqueeze(0)), case.module(case.x.unsqueeze(0)))


def test_symmetric_branch_runs():
    torch.manual_seed(0)
    K, N, M = 256, 64, 16
    lin = torch.nn.Linear(K, N, bias=False)
    w = torch.randint(-7, 8, (N, K)).half()
    mod = MixedQLinear.from_float(lin, w, torch.ones(N, 1), fp_indices=None, symm=True, bits=4).to(dev())
    x = torch.randn(M, K).half().to(dev())
    out = mod(x.unsqueeze(0))[0].cpu()
    qs = (x.abs().max(1)[0].unsqueeze(1) / (1 << (4 - 1) - 1)).half().cpu()
    q = kp.sym_quantize(x.cpu(), qs, 4)
    acc = kp.int4_matmul(q, kp.pack_to_i4(w.to(torch.int8)))
    ref = kp.sym_dequantize(acc, qs, torch.ones(1, N).half(), torch.zeros(M, N).half(), 32)
    assert torch.equal(out, ref)


@pytest.mark.parametrize("bits,K,F", [(4, 4352, 256), (8, 2304, 256)])
def test_engines_agree_on_the_same_rows_across_token_counts(bits, K, F):
    """16, 128 and 129 tokens take three different engines (mma.sync streaming, tcgen05 streaming, tiled tcgen05
    GEMM).  The integer part is exact in all of them; the tiled engine rounds (outlier product + bias) to the storage
    type before the dequantize step (as the reference's F.linear output is rounded, experiments/qlinear.py:124) while
    the streaming engines keep it in fp32, so the same token differs by at most a couple of units in the last place of
    the largest outputs: 5e-3 of the output RMS in fp16."""
    N = 520
    case = make_layer("t", 129, K, N, bits, F=F, seed=11, device=dev(), clip=False)
    outs = {}
    for M in (16, 128, 129):
        outs[M] = case.module(case.x[:M].contiguous().unsqueeze(0))[0]
    assert_device_clean()
    ref = _oracle_out(case, round_y=False)
    for M, out in outs.items():
        assert rel_rms_err(out.cpu(), ref[:M]) < TOL_RMS, M
    assert rel_rms_err(outs[128][:16], outs[16]) < 5e-3
    assert rel_rms_err(outs[129][:128], outs[128]) < 5e-3


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs 2 GPUs")
def test_layers_on_two_devices_of_one_process():
    """One process driving layers on cuda:0 and cuda:1 in turn (the reference's llama_multigpu places layers this way,
    experiments/llama.py:295-326): shared-memory opt-ins and occupancy answers are kept per device.  Plain launches,
    no peer memory."""
    outs = []
    for d in (0, 1, 0, 1):
        device = torch.device("cuda", d)
        for M in (16, 300):
            case = make_layer("t", M, 1088, 520, 4, F=64, seed=5, device=device, clip=False)
            out = case.module(case.x.unsqueeze(0))
            torch.cuda.synchronize(device)
            assert out.device == device
            assert rel_rms_err(out[0].cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
            with torch.cuda.device(device):
                assert _lib.device_status() == 0
            outs.append((M, out[0].cpu()))
    assert torch.equal(outs[0][1], outs[2][1]) and torch.equal(outs[1][1], outs[3][1])      # cuda:0 == cuda:1


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,F,bits", [(1, 1024, 264, 64, 4), (16, 1024, 264, 0, 8), (17, 1024, 264, 64, 4), (128, 1024, 130, 64, 4),
                                          (129, 1024, 264, 64, 4), (300, 1024, 261, 32, 8), (9, 112, 24, 32, 4)])
def test_single_native_call_equals_quantizer_and_layer_calls(M, K, N, F, bits, dtype):
    """A layer without a shared input runs quantizer and fused kernel from one native call: same bits as the two calls of a
    shared input, for matrices and batches of one, with the settings that send few tokens to the tensor-core GEMM, into a
    caller's buffer; and it refuses what they refuse."""
    case = make_layer("t", M, K, N, bits, F=F, seed=3, device=dev(), dtype=dtype, clip=False)
    layer, x = case.module, case.x
    one = layer(x)
    assert one.shape == (1, M, N) and torch.equal(layer(x.unsqueeze(0)), one)
    assert torch.equal(layer(torch.stack([x, x + 1])), one)               # a batch: its first matrix
    layer.shared_input = SharedQuantizedInput(1)
    assert torch.equal(layer(x), one)
    layer.shared_input = None
    try:
        _lib.set_small_m(False)
        off = layer(x)
        layer.shared_input = SharedQuantizedInput(1)
        assert torch.equal(layer(x), off)
    finally:
        _lib.set_small_m(True)
        layer.shared_input = None
    buf = torch.full((M, N + 8), -1.0, dtype=dtype, device=dev())
    layer.out_buffer = buf[:, :N]
    assert layer(x).data_ptr() == buf.data_ptr() and torch.equal(buf[:, :N], one[0]) and (buf[:, N:] == -1).all()
    layer.out_buffer = None
    assert layer(x[:0]).shape == (1, 0, N)
    for bad, why in ((x[:, :-2].contiguous(), "column counts"), (x.float(), "float16 or bfloat16")):
        with pytest.raises(RuntimeError, match=why):
            layer(bad)
    if M > 1:                                                             # the right shape at a wider pitch
        with pytest.raises(RuntimeError, match="to be contiguous"):
            layer(torch.nn.functional.pad(x, (0, 8))[:, :K])
    assert torch.equal(layer(x), one)
    assert_device_clean()


@pytest.mark.parametrize("K,N,F,bits", [(1088, 130, 64, 4), (4352, 512, 256, 4), (608, 264, 0, 8), (11264, 512, 256, 8)],
                         ids=["int4", "int4_split", "int8", "int8_split"])
@pytest.mark.parametrize("M", [17, 31, 33, 48, 64, 65, 80, 97, 112, 128])
def test_streaming_engine_at_every_width(M, K, N, F, bits):
    """The tcgen05 streaming engine pads the tokens to the next multiple of 16 and plans shared and tensor memory for that
    width (two CTAs per SM up to 64); K whole or split over a cluster whose CTAs each finish a share of the tokens."""
    case = make_layer("t", M, K, N, bits, F=F, seed=M, device=dev(), clip=False)
    out = case.module(case.x.unsqueeze(0))[0]
    assert rel_rms_err(out.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
    assert torch.equal(case.module(case.x.unsqueeze(0))[0], out)
    few = case.module(case.x[:16].contiguous())[0]                       # other engine: exact integers, fp32 outlier product
    assert rel_rms_err(out[:16].cpu(), few.cpu()) < 5e-3
    assert_device_clean()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("engine", [_lib.ENGINE_TCGEN05, _lib.ENGINE_TCGEN05_TS], ids=["smem_operands", "tmem_operand"])
@pytest.mark.parametrize("N", [3600, 3599, 3602])
@pytest.mark.parametrize("F", [64, 0])
def test_many_tiles_per_cta_and_ragged_rows(N, F, engine, dtype):
    """Four tiles of 32 columns per CTA or pair, so that both accumulator regions change hands several times, with integer
    products of one and of three k-blocks; output rows with 16-byte, 2-byte and 4-byte alignment, the last tile ragged in
    both directions."""
    for K in (64 + F, 320 + F):
        case = make_layer("t", 300, K, N, 4, F=F, seed=N, device=dev(), dtype=dtype, clip=False)
        try:
            _lib.set_engine(engine)
            _lib.set_tile_n(32)
            for pair in (2, 1):
                _lib.set_cta_pair(pair)
                out = case.module(case.x.unsqueeze(0))[0]
                assert rel_rms_err(out.cpu(), _oracle_out(case, round_y=True)) < (TOL_RMS if dtype == torch.float16 else 4e-2)
        finally:
            _lib.set_engine(_lib.ENGINE_AUTO)
            _lib.set_tile_n(0)
            _lib.set_cta_pair(0)
    assert_device_clean()


@pytest.mark.parametrize("M,K,N,F,bits", [(5, 1088, 1000, 64, 4), (17, 4352, 4096, 256, 4), (64, 4352, 4096, 256, 4), (128, 4352, 4096, 256, 4),
                                          (100, 2304, 1000, 256, 8), (300, 1088, 1000, 64, 4)])
def test_weights_written_on_the_same_stream_are_seen(M, K, N, F, bits):
    """Weights are an argument of the fused launch: integer and outlier weights that a kernel writes on the stream directly
    before it, with nothing in between, are the ones that are used, although the launch overlaps its predecessor; the same
    through the module after an in-place update.  (The ring engine for few tokens asks for settled weights.)"""
    case = make_layer("t", M, K, N, bits, F=F, seed=M, device=dev(), clip=False)
    layer = case.module
    w0, f0 = layer.int_weight.clone(), layer.fp_weight.clone()
    layer.shared_input = SharedQuantizedInput(1 << 30)            # quantized once: the launches below stand alone
    layer(case.x)

    def update(flip):
        torch.bitwise_xor(w0, 0x11 if flip else 0, out=layer.int_weight)
        torch.mul(f0, -1 if flip else 1, out=layer.fp_weight)

    want = []
    try:
        _lib.set_pdl(False)
        for flip in (0, 1):
            update(flip)
            want.append(layer(case.x).clone())
    finally:
        _lib.set_pdl(True)
    assert not torch.equal(*want)
    torch.cuda.synchronize()
    got = []
    for rep in range(12):
        update(rep & 1)
        got.append(layer(case.x))
    layer.shared_input = None
    for rep in range(6):
        update(rep & 1)
        got.append(layer(case.x))
    torch.cuda.synchronize()
    for rep, out in enumerate(got):
        assert torch.equal(out, want[rep & 1]), rep
    assert_device_clean()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("M,bits", [(16, 4), (3, 8), (128, 4)])
def test_few_tokens_after_an_in_place_update_of_the_weights(M, bits, shared):
    """The module directly after in-place updates of its weights by kernels of the same stream, at sizes where few tokens go
    to the ring engine, which reads weights ahead of the stream's earlier launches (16 MiB packed, 32 MiB int8): the results
    are those of plain stream order; so are a call without an update in between and one captured together with its update."""
    case = make_layer("t", M, 4096 + 64, 8192, bits, F=64, seed=M, device=dev(), clip=False)
    layer, x = case.module, case.x
    w0, f0 = layer.int_weight.clone(), layer.fp_weight.clone()
    layer.shared_input = SharedQuantizedInput(1) if shared else None

    def update(flip):
        torch.mul(f0, -1 if flip else 1, out=layer.fp_weight)
        torch.bitwise_xor(w0, 0x11 if flip else 0, out=layer.int_weight)

    want = []
    try:
        _lib.set_pdl(False)
        for flip in (0, 1):
            update(flip)
            want.append(layer(x).clone())
    finally:
        _lib.set_pdl(True)
    torch.cuda.synchronize()
    got = []
    for rep in range(8):
        update(rep & 1)
        got.append((layer(x), layer(x)))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            update(0)
            a = layer(x)
            update(1)
            b = layer(x)
        for _ in range(3):
            g.replay()
    torch.cuda.synchronize()
    for rep, pair in enumerate(got):
        assert all(torch.equal(out, want[rep & 1]) for out in pair), rep
    assert torch.equal(a, want[0]) and torch.equal(b, want[1])
    assert_device_clean()


@pytest.mark.parametrize("N,bits", [(8192, 4), (1000, 4), (8192, 8)])
def test_ring_engine_settings_give_the_same_bits(N, bits):
    """The ring engine with its weights loaded before or after the wait, or also asked of L2, and with either ring depth."""
    case = make_layer("t", 16, 4096 + 64, N, bits, F=64, seed=N, device=dev(), clip=False)
    try:
        _lib.set_small_m(_lib.SMALL_M_TMA_MMA)
        want = case.module(case.x)
        for key, values in ((_lib.CFG_STREAM_PRELOAD, (0, 2, 1)), (_lib.CFG_STREAM_RING, (0, 1, 2))):
            for v in values:
                _lib.check(_lib.load().quik_config_set(key, v), "quik_config_set")
                for _ in range(3):
                    assert torch.equal(case.module(case.x), want)
    finally:
        _lib.set_small_m(True)
        _lib.check(_lib.load().quik_config_set(_lib.CFG_STREAM_PRELOAD, 1), "quik_config_set")
        _lib.check(_lib.load().quik_config_set(_lib.CFG_STREAM_RING, 2), "quik_config_set")
    assert_device_clean()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("slabs,K,F", [(1, 96, 64), (3, 160, 0), (2, 352, 64), (15, 2304, 64), (16, 2304, 64), (34, 2304, 64), (70, 1088, 64),
                                       (74, 2304, 64), (75, 4352, 256), (96, 5632, 64), (149, 1088, 64)])
def test_streaming_engine_splits_and_short_sums(slabs, K, F, bits):
    """One to a few integer blocks (the two int8 issuing warps then have none, one or several each), and numbers of 128-row slabs on
    both sides of every line of the rule for splits and CTAs per SM.  The sums are integers: the rows of a call equal those of
    a call for other token counts, which run another split, another plan or (up to 16 tokens) another engine, up to the
    place of the rounding; the smallest layers are compared with the oracle."""
    N = 128 * slabs - 5
    case = make_layer("t", 128, K, N, bits, F=F, seed=slabs, device=dev(), clip=False)
    ref = case.module(case.x)[0]
    if slabs <= 16:
        assert rel_rms_err(ref.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
    few = case.module(case.x[:16].contiguous())[0]
    assert rel_rms_err(ref[:16].cpu(), few.cpu()) < 5e-3
    for M in (17, 32, 33, 64, 65, 97):
        out = case.module(case.x[:M].contiguous())[0]
        assert torch.equal(case.module(case.x[:M].contiguous())[0], out)
        assert rel_rms_err(out.cpu(), ref[:M].cpu()) < 5e-3
    assert_device_clean()


@pytest.mark.parametrize("M,slabs,K,F", [(80, 149, 2560, 64), (128, 149, 2560, 64), (65, 222, 5152, 0), (97, 300, 2560, 64),
                                         (33, 297, 2560, 64), (17, 444, 5152, 0)])
def test_streaming_engine_beyond_a_full_wave(M, slabs, K, F):
    """More slabs of 128 rows than run at once: the last ones are a launch of their own that splits K.  One slab beyond a wave up to
    half a wave, two CTAs per SM up to 64 tokens, with the last slab ragged, into a window of a wider matrix."""
    N = 128 * slabs - 5
    case = make_layer("t", M, K, N, 4, F=F, seed=M, device=dev(), clip=False)
    out = case.module(case.x.unsqueeze(0))[0]
    assert rel_rms_err(out.cpu(), _oracle_out(case, round_y=False)) < TOL_RMS
    slab = torch.full((M, N + 7), -1234.0, dtype=torch.float16, device=dev())
    case.module.out_buffer = slab[:, 3:3 + N]
    case.module(case.x.unsqueeze(0))
    case.module.out_buffer = None
    assert torch.equal(slab[:, 3:3 + N], out)
    slab[:, 3:3 + N] = -1234.0
    assert bool((slab == -1234.0).all())
    assert_device_clean()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("M,bits,F", [(5, 4, 64), (40, 4, 64), (200, 4, 64), (200, 8, 0)])
def test_native_path_follows_the_buffers(M, bits, F, shared):
    """The native host path works from operands derived from the layer's buffers: after each change of a buffer, in place or by
    another tensor, a call gives the bits of the path that derives them anew, and so does a copy of the layer."""
    case = make_layer("t", M, 1024 + F, 264, bits, F=F, seed=M, device=dev(), clip=False)
    layer, x = case.module, case.x.unsqueeze(0)
    layer.shared_input = SharedQuantizedInput(1) if shared else None

    def check():
        want = layer._forward_checked(x)
        assert layer._plan is not None
        got = layer(x)
        assert torch.equal(got, want)
        return got

    first = check()
    assert torch.equal(copy.deepcopy(layer)(x), first)
    with torch.no_grad():
        ids = layer.int_indices.clone()
        layer.int_indices[0], layer.int_indices[1] = ids[1], ids[0]                    # in place
        got = layer(x)
        assert not torch.equal(got, first) and torch.equal(got, layer._forward_checked(x))
        layer.int_indices = ids                                                       # another tensor
        assert torch.equal(layer(x), first)
        check()
        layer.int_weight.copy_(layer.int_weight.flip(0))
        got = layer(x)
        assert torch.equal(got, layer._forward_checked(x)) and not torch.equal(got, first)
        layer.weights_scales = layer.weights_scales * 2
        layer.bias = None
        check()
    with pytest.raises(Exception):
        layer(x.cpu())
    assert_device_clean()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("M,bits", [(5, 4), (200, 4), (200, 8)])
def test_buffers_replaced_at_the_same_address(M, bits, shared):
    """A buffer that is replaced by another tensor at the same address and version (memory that the allocator gives out again): the
    next call uses the new one's contents."""
    case = make_layer("t", M, 1024 + 64, 264, bits, F=64, seed=M, device=dev(), clip=False)
    layer, x = case.module, case.x.unsqueeze(0)
    layer.shared_input = SharedQuantizedInput(1) if shared else None
    for name in ("int_weight", "int_indices", "fp_indices"):
        old = getattr(layer, name).clone()
        memory = old.clone()
        setattr(layer, name, memory.data)                     # .data: another tensor over the memory, at version 0
        layer(x)
        first = layer(x)
        at = getattr(layer, name).data_ptr(), getattr(layer, name)._version
        memory.copy_(old.flip(0))
        setattr(layer, name, memory.data)
        assert (getattr(layer, name).data_ptr(), getattr(layer, name)._version) == at
        got = layer(x)
        assert torch.equal(got, copy.deepcopy(layer)(x)) and not torch.equal(got, first)
        setattr(layer, name, old)
        assert torch.equal(layer(x), first)
    assert_device_clean()


@pytest.mark.parametrize("M,bits", [(5, 4), (40, 4), (200, 4), (200, 8)])
def test_members_that_never_quantize_need_no_ids(M, bits):
    """A group of three on one quantized input: only the member that quantizes derives column ids; the others may have none, at the
    first call and at later ones.  One that quantizes later derives its own then, and its next calls take the native path too."""
    case = make_layer("t", M, 1024 + 64, 264, bits, F=64, seed=M, device=dev(), clip=False)
    x = case.x.unsqueeze(0)
    want = case.module(x)
    shared = SharedQuantizedInput(3)
    a, b, c = (copy.deepcopy(case.module) for _ in range(3))
    for m in (a, b, c):
        m.shared_input = shared
    ids, fp_ids = b.int_indices.clone(), b.fp_indices.clone()
    for m in (b, c):
        m.int_indices.zero_()
        m.fp_indices.zero_()
    for _ in range(3):
        for m in (a, b, c):
            assert torch.equal(m(x), want)
            assert m._plan is not None and (m._plan[0] is None) == (m is not a) and ("int16" in m._cache) == (m is a)
    with pytest.raises(RuntimeError, match="exactly once"):
        b(x)
    assert shared.qint_x is None and shared.cur_group_elem == 0
    b.int_indices.copy_(ids)
    b.fp_indices.copy_(fp_ids)
    for _ in range(2):
        for m in (b, c, a):
            assert torch.equal(m(x), want)
    assert b._plan[0] is not None and c._plan[0] is None
    norm = torch.ones(x.shape[-1], dtype=x.dtype, device=x.device)
    c.int_indices.copy_(ids)
    c.fp_indices.copy_(fp_ids)
    got = []
    for _ in range(3):
        c.quantize_rmsnorm(x, norm, 1e-5)
        got.append([m(x) for m in (c, a, b)])
    assert c._plan[0] is not None
    assert all(torch.equal(t, got[0][0]) for outs in got for t in outs) and not torch.equal(got[0][0], want)
    assert_device_clean()


@pytest.mark.parametrize("F", [0, 64])
def test_quantized_weights_at_a_reused_address_are_waited_for(F):
    """Few tokens through the ring engine, which loads its weights before it waits for the stream: weights that the quantizer (which
    lets later launches start early) has just written, in a tensor at the address and version of the last ones."""
    M, K, N = 16, 4096 + F, 8192
    case = make_layer("t", M, K, N, 8, F=F, seed=F, device=dev(), clip=False)
    layer, x = case.module, case.x.unsqueeze(0)
    memory = layer.int_weight.clone()
    g = torch.Generator().manual_seed(7)
    sources = [torch.randn(N, K - F, generator=g).half().to(dev()) for _ in range(2)]
    all_ids, meta = torch.arange(K - F, device=dev()), torch.empty(2 * N, dtype=torch.float16, device=dev())

    def write(i):
        _lib.check(_lib.load().quik_asym_quantize(_lib.ptr(sources[i]), 0, N, K - F, _lib.ptr(all_ids), K - F, None, 0, 8,
                                                  _lib.ptr(memory), _lib.ptr(meta), None, _lib.stream_of(memory)), "quantize")
        layer.int_weight = memory.data
    want = []
    for i in (0, 1):
        write(i)
        torch.cuda.synchronize()
        want.append(layer(x).clone())
    assert not torch.equal(*want)
    for rep in range(20):
        write(rep & 1)
        assert torch.equal(layer(x), want[rep & 1]), rep
    assert_device_clean()


def test_plans_only_where_they_can_serve():
    """A plan goes with the layer's cache, and there is none for calls that the native path declines: a bias or weights that are no
    buffers, an output buffer of the caller.  Outputs are the same either way."""
    case = make_layer("t", 200, 1024 + 64, 264, 4, F=64, seed=3, device=dev(), clip=False)
    layer, x = case.module, case.x.unsqueeze(0)
    layer.bias = None
    want = layer(x)
    w8 = weakref.ref(layer._plan[2])
    layer._cache.clear()
    assert layer._plan is None and w8() is None
    assert torch.equal(layer(x), want) and layer._plan is not None
    layer.out_buffer = torch.empty_like(want[0])
    assert torch.equal(layer(x), want) and layer._plan is None
    layer.out_buffer = None
    assert torch.equal(layer(x), want) and layer._plan is not None
    for name in ("bias", "fp_weight", "reduced_w"):
        value = layer._buffers.pop(name)
        object.__setattr__(layer, name, value)
        for _ in range(2):
            assert torch.equal(layer(x), want) and layer._plan is None
        object.__delattr__(layer, name)
        layer.register_buffer(name, value)
        assert torch.equal(layer(x), want) and layer._plan is not None
    assert_device_clean()


@pytest.mark.parametrize("writer", ["unpack", "dequantize", "rotary"])
def test_operators_before_a_launch_settle_its_weights(writer):
    """The ring engine loads its weights before it waits for the stream.  Weights that the widening, dequantize or rotary operator has
    just written are used as written: nothing starts before those operators are complete (calls of the C interface, which has no
    record of weights)."""
    M, F, N = 16, 64, 8192
    K = 4096 + F
    case = make_layer("t", M, K, N, 8, F=F, seed=5, device=dev(), clip=False)
    layer, lib = case.module, _lib.load()
    i16, f16 = layer._idx16()
    w, fw, p, st = layer.int_weight.clone(), layer.fp_weight.clone(), _lib.ptr, _lib.stream_of(case.x)
    q, meta = torch.empty(M, K - F, dtype=torch.int8, device=dev()), torch.empty(2 * M, dtype=torch.float16, device=dev())
    fp_x, out = torch.empty(M, F, dtype=torch.float16, device=dev()), torch.empty(M, N, dtype=torch.float16, device=dev())
    packed = [torch.randint(0, 256, (N, (K - F) // 2), dtype=torch.uint8, device=dev()) for _ in range(2)]
    acc = [torch.randint(-99, 99, (N, F), dtype=torch.int32, device=dev()) for _ in range(2)]
    ones, zeros = torch.ones(2 * N, dtype=torch.float16, device=dev()), torch.zeros(N * F, dtype=torch.float16, device=dev())
    quarter = [torch.tensor(v, dtype=torch.float16, device=dev()).expand(N, F // 2).contiguous() for v in (0.0, 1.0)]

    def write(i):
        if writer == "unpack":
            rc = lib.quik_unpack_int4(p(packed[i]), p(w), N, K - F, st)
        elif writer == "dequantize":
            rc = lib.quik_asym_dequantize(p(acc[i]), p(ones), p(ones), p(zeros), p(zeros), p(fw), 0, N, F, 8, st)
        else:                                             # a quarter turn of every pair of columns
            rc = lib.quik_rotary_inplace(p(fw), None, p(quarter[0]), p(quarter[1]), 0, N, 1, 0, F, st)
        _lib.check(rc, writer)

    def launch():
        _lib.check(lib.quik_layer_quantize(0, p(case.x), None, 0.0, 0, M, K, p(i16), K - F, p(f16), F, 8, 1, 1, p(q), p(meta), p(fp_x), st),
                   "quantize")
        _lib.check(lib.quik_mixed_linear(p(q), 0, p(w), 0, p(meta), p(layer.weights_scales), p(layer.reduced_w), p(fp_x), p(fw), None,
                                         p(out), 0, M, N, K - F, F, 8, st), "linear")
        return out.clone()
    want = []
    for i in range(4):                                    # (four quarter turns come back to the start)
        write(i & 1)
        torch.cuda.synchronize()
        want.append(launch())
    assert not torch.equal(want[0], want[1])
    for rep in range(40):
        write(rep & 1)
        assert torch.equal(launch(), want[rep % 4]), rep
    assert_device_clean()


@pytest.mark.parametrize("M,slabs,K_int,F,bits,split", [
    (80, 149, 4096, 0, 4, 8), (80, 222, 4096, 64, 4, 2), (80, 222, 3840, 64, 4, 0), (80, 223, 8192, 0, 4, 0), (80, 149, 2048, 64, 4, 0),
    (128, 178, 2816, 64, 8, 4), (128, 178, 2688, 64, 8, 0), (80, 445, 4864, 0, 4, 8), (80, 445, 4608, 0, 4, 0),
    (40, 370, 10240, 0, 4, 2), (40, 370, 9984, 0, 4, 0), (40, 371, 10240, 0, 4, 0), (64, 300, 6144, 64, 4, 8), (64, 300, 4608, 64, 4, 0),
    (20, 370, 8192, 0, 8, 2), (20, 370, 8064, 0, 8, 0)])
def test_streaming_engine_second_launch_is_chosen_by_what_it_saves(M, slabs, K_int, F, bits, split):
    """Slabs beyond full waves split K in a launch of their own where that takes enough blocks out of the chain, up to a quarter of a
    wave with two CTAs per SM, and for more blocks from three full waves on; both sides of each line.  The first CTA of the last launch counts its blocks: all of the layer's (split 0),
    or its share.  The outputs are those of the tiled engine."""
    N, d = 128 * slabs - 3, dev()
    layer = MixedQLinear(K_int + F, 8, fp_features_num=F, bits=bits).to(d)
    g = torch.Generator(device=d).manual_seed(slabs)
    layer.out_features = N
    if bits == 4:
        layer.int_weight = torch.randint(0, 256, (N, K_int // 2), dtype=torch.uint8, device=d, generator=g)
    else:
        layer.int_weight = torch.randint(-128, 128, (N, K_int), dtype=torch.int8, device=d, generator=g)
    layer.weights_scales = 0.01 + 0.01 * torch.rand(N, 1, device=d, generator=g).half()
    layer.reduced_w = torch.randn(1, N, device=d, generator=g).half()
    layer.bias = torch.randn(N, device=d, generator=g).half()
    layer.int_indices, layer.fp_indices = torch.arange(K_int, device=d), torch.arange(K_int, K_int + F, device=d)
    if F:
        layer.fp_weight = torch.randn(N, F, device=d, generator=g).half()
    x = torch.randn(1, M, K_int + F, device=d, generator=g).half()
    counters = torch.zeros(16 * 1024, dtype=torch.int64, device=d)
    try:
        _lib.check(_lib.load().quik_debug_counters(counters.data_ptr()), "quik_debug_counters")
        out = layer(x)
        torch.cuda.synchronize()
    finally:
        _lib.load().quik_debug_counters(None)
    total = K_int * bits // 1024 + F // 64
    assert int(counters[3]) == (total // split if split else total)
    try:
        _lib.set_small_m(_lib.SMALL_M_OFF)
        want = layer(x)
    finally:
        _lib.set_small_m(True)
    assert rel_rms_err(out.cpu(), want.cpu()) < 5e-3
    assert_device_clean()
