"""GPU parity tests of the tensor-core dequant-GEMM (tcgen05 / TMEM path), through the C ABI.

The GEMM takes 16-bit activations (the benchmark's prefill configuration: bf16 in, fp32 accumulate) and
feeds the tensor cores fp16 weights: w = scale*q + bias rounded once to fp16, a relative error of at most
2^-12 per weight, random in sign.  The oracle sees the same rounded activations, so what is compared is
that weight rounding plus the fp32 accumulation order.  Bars:

* benchmark value distributions (|w| ~ 0.01, |y| < 1): max |got-ref| / max(1,|ref|) < 1e-3 and normwise
  ||got-ref|| / ||ref|| < 1e-3;
* the reference fixture's much larger magnitudes (|w| ~ 0.3, |y| ~ 5-20): normwise < 5e-4 (= 2 * 2^-12);
  the element-wise metric, which divides the absolute error by max(1,|ref|) even where |ref| is small
  next to the row's terms, must stay < 1.5e-2.  (fp32 activations never take this path: they, and all
  other widths, take the full-precision GEMM, whose bars stand with its tests.)"""
import importlib

import numpy as np
import pytest
import torch

from helpers import DevLayer, as_dtype, run

pytestmark = pytest.mark.gpu

synth = importlib.import_module("mlx-runner_b200.synth")


def _ref(oracle, lay_or_fx, x_rounded, K, bits, gs, sdt, bias=None):
    return oracle.qmatmul(lay_or_fx.packed, lay_or_fx.scales_raw, lay_or_fx.biases_raw, sdt, x_rounded, K, bits, gs, bias=bias)


@pytest.mark.parametrize("x_dtype", [1, 2])
def test_gemm_is_selected_and_matches_oracle(mlxq, oracle, x_dtype):
    # one full tile, bf16 scales: fp16 operands hold the weights almost exactly
    O, K, T = 256, 512, 128
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, scale_type=oracle.BF16, seed=5)
    layer = DevLayer.from_fixture(mlxq, fx)
    assert layer.linear.kernelFor(T, x_dtype, 0) == "qgemm"
    assert layer.linear.gemmTileTokens(T) == 128 and layer.linear.gemmTileTokens(4) == 0
    assert layer.linear.gemmTileTokens(129) == 256          # longer batches take the 128-row x 256-token tile
    x = oracle.RNG(77).floats(T * K).reshape(T, K)
    xr = as_dtype(x, x_dtype).float().cpu().numpy()
    got = run(layer, x, T, x_dtype=x_dtype)
    mlxq.streamStatus(None, 0)
    ref = fx.reference(xr)
    nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
    assert nrm < 5e-4 and oracle.max_rel_err(got, ref) < 1.5e-2, f"x dtype {x_dtype}: normwise {nrm}"


@pytest.mark.parametrize("T,O,K,gs", [(17, 40, 512, 32), (33, 41, 576, 64), (517, 520, 576, 32), (96, 2050, 1024, 128),
                                      (300, 777, 4096, 64)])
def test_gemm_ragged_shapes(mlxq, oracle, T, O, K, gs):
    # tokens and rows that do not fill a tile, strided x / y with NaN padding, row bias, bf16 output too
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=gs, scale_type=oracle.BF16, with_bias=True, seed=T + O)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = oracle.RNG(T * 7 + 4).floats(T * K).reshape(T, K)
    xr = as_dtype(x, 2).float().cpu().numpy()
    ref = _ref(oracle, fx, xr, K, 4, gs, oracle.BF16, bias=fx.bias)
    assert layer.linear.kernelFor(T, 2, 0) == "qgemm"
    got = run(layer, x, T, x_dtype=2, x_stride=K + 8, y_stride=O + 3)
    nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
    assert nrm < 5e-4 and oracle.max_rel_err(got, ref) < 1.5e-2, f"normwise {nrm}"
    got16 = run(layer, x, T, x_dtype=2, y_dtype=2, y_stride=O + 5)
    assert float(np.linalg.norm(got16 - ref) / np.linalg.norm(ref)) < 4e-3        # bf16 output rounding, 2^-9 per element
    mlxq.streamStatus(None, 0)


def test_gemm_baseline_distribution_fp16_scales(mlxq, oracle):
    # the prefill configuration's value distribution at reduced O (oracle cost), fp16 and bf16 scales
    O, K, T = 512, 4096, 256
    for sdt in (synth.F16, synth.BF16):
        lay = synth.make_layer(O, K, 4, 64, sdt, seed=9, bias_noise=True)
        layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, sdt, K)
        _, x = synth.make_activations(T, K, synth.BF16, seed=2)
        ref = oracle.qmatmul(lay.packed, lay.scales_raw, lay.biases_raw, sdt, x, K, 4, 64)
        got = run(layer, x, T, x_dtype=2)
        err = oracle.max_rel_err(got, ref)
        nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
        assert err < 1e-3 and nrm < 1e-3, f"scales {sdt}: max-rel {err}, normwise {nrm}"


def test_gemm_fp16_scales_reference_fixture_magnitudes(mlxq, oracle):
    O, K, T = 384, 1024, 160
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, scale_type=oracle.F16, seed=12)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = oracle.RNG(13).floats(T * K).reshape(T, K)
    xr = as_dtype(x, 1).float().cpu().numpy()
    ref = fx.reference(xr)
    got = run(layer, x, T, x_dtype=1)
    nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
    assert nrm < 5e-4 and oracle.max_rel_err(got, ref) < 1.5e-2


def test_gemm_token_outputs_do_not_depend_on_the_batch(mlxq, oracle):
    # KernelTests.swift:168-184 for the GEMM family: bit-identical rows whatever batch they ride in
    O, K = 2050, 1024
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, seed=3)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = oracle.RNG(11).floats(256 * K).reshape(256, K)
    full = run(layer, x, 256, x_dtype=2).view(np.uint32)
    for T in (17, 33, 96, 131):
        assert np.array_equal(run(layer, x[:T], T, x_dtype=2).view(np.uint32), full[:T]), f"T {T} vs T 256"


def test_gemm_round_trip_property_at_full_size(mlxq, oracle):
    # full prefill size (14336 x 4096, M = 2048): linearity in x, checked without the oracle --
    # W.(x1 + x2) = W.x1 + W.x2 for activations whose sum is exact in bf16 -- plus an oracle check on a
    # random sample of output rows.
    O, K, T = 14336, 4096, 2048
    lay = synth.make_layer(O, K, 4, 64, synth.BF16, seed=21, keep_codes=False)
    layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, synth.BF16, K)
    g = np.random.default_rng(5)
    x1 = g.integers(-8, 9, size=(T, K)).astype(np.float32) / 8       # small dyadic values: sums stay exact in bf16
    x2 = g.integers(-8, 9, size=(T, K)).astype(np.float32) / 8
    y1, y2, y12 = run(layer, x1, T, x_dtype=2), run(layer, x2, T, x_dtype=2), run(layer, x1 + x2, T, x_dtype=2)
    assert oracle.max_rel_err(y12, y1 + y2) < 1e-4
    rows = np.sort(g.choice(O, size=64, replace=False))
    sub = oracle.qmatmul(lay.packed[rows], lay.scales_raw[rows], lay.biases_raw[rows], synth.BF16, x1[:128], K, 4, 64)
    assert oracle.max_rel_err(y1[:128][:, rows], sub) < 1e-3
    mlxq.streamStatus(None, 0)


def test_gemm_repeats_bit_for_bit_at_full_size(mlxq):
    # 14336 x 4096, M = 2048, twelve calls on the same inputs: the pipeline's hand-offs (TMA rings, tensor-memory A
    # ring, deferred epilogue) leave no room for timing to change a single bit.  Tensor-memory stores issued after the
    # lanes of a warp had polled a barrier one by one showed up here as a few rows of one tile differing.
    O, K, T = 14336, 4096, 2048
    lay = synth.make_layer(O, K, 4, 64, synth.BF16, seed=31, keep_codes=False)
    layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, synth.BF16, K)
    _, xv = synth.make_activations(T, K, synth.BF16, seed=100)
    x = torch.from_numpy(xv).to("cuda").to(torch.bfloat16)
    ys = [torch.empty((T, O), dtype=torch.float32, device="cuda") for _ in range(2)]
    layer.linear.encode(None, x, K, ys[0], O, T)
    for call in range(12):
        layer.linear.encode(None, x, K, ys[1], O, T)
        torch.cuda.synchronize()
        differing = int((ys[1].view(torch.int32) != ys[0].view(torch.int32)).sum())
        assert differing == 0, f"call {call}: {differing} outputs differ from the first call's"
    mlxq.streamStatus(None, 0)


def _bf16_bits(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.int64)


@pytest.mark.parametrize("O,K", [(14336, 4096), (4096, 14336)])
def test_gemm_prefill_sizes_against_oracle(mlxq, oracle, O, K):
    # the prefill configuration at its own sizes: M = 128, 512, 8192 on both orientations (M = 2048 is covered above);
    # the oracle on a sample of rows x tokens.  fp32 output: the 1e-3 bar.  bf16 output: within one bf16 ulp of the
    # oracle rounded to bf16 (outputs so close to zero that an ulp is below the fp32 bar are held to that bar instead).
    lay = synth.make_layer(O, K, 4, 64, synth.BF16, seed=O % 97, keep_codes=False)
    layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, synth.BF16, K)
    g = np.random.default_rng(K)
    rows = np.sort(g.choice(O, size=48, replace=False))
    for T in (128, 512, 8192):
        _, x = synth.make_activations(T, K, synth.BF16, seed=T)
        toks = np.sort(np.concatenate([np.arange(8), g.choice(np.arange(8, T), size=24, replace=False)]))
        ref = oracle.qmatmul(lay.packed[rows], lay.scales_raw[rows], lay.biases_raw[rows], synth.BF16, x[toks], K, 4, 64)
        assert layer.linear.kernelFor(T, 2, 0) == "qgemm"
        got = run(layer, x, T, x_dtype=2)[toks][:, rows]
        err = oracle.max_rel_err(got, ref)
        assert err < 1e-3, f"{O}x{K} T={T}: max relative error {err}"
        got16 = run(layer, x, T, x_dtype=2, y_dtype=2)[toks][:, rows]
        ulps = np.abs(_bf16_bits(got16) - _bf16_bits(ref))
        near_zero = np.abs(got16 - ref) <= 1e-3 * np.maximum(1.0, np.abs(ref))
        assert np.all((ulps <= 1) | near_zero), f"{O}x{K} T={T}: bf16 output off by {int(ulps[~near_zero].max())} ulps"
    mlxq.streamStatus(None, 0)


def test_prepared_table_changes_nothing(mlxq, oracle):
    # mlxq_linear_prepare builds the GEMM's scale/bias table ahead; a batch encoded while its stream is being captured
    # cannot keep a table and stages it per call.  All routes must give the same bits.
    O, K, T = 768, 2048, 160
    lay = synth.make_layer(O, K, 4, 64, synth.BF16, seed=77, bias_noise=True)
    _, xv = synth.make_activations(T, K, synth.BF16, seed=5)
    x = torch.from_numpy(xv).to("cuda").to(torch.bfloat16)
    outs = []
    for route in ("prepared", "first call builds it", "captured"):
        layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, synth.BF16, K, name=route)
        y = torch.full((T, O), float("nan"), dtype=torch.float32, device="cuda")
        if route == "prepared":
            layer.linear.prepare(None)
        if route == "captured":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                layer.linear.encode(torch.cuda.current_stream(), x, K, y, O, T)
            g.replay()
        else:
            layer.linear.encode(None, x, K, y, O, T)
        torch.cuda.synchronize()
        mlxq.streamStatus(None, 0)
        outs.append(y.cpu().numpy())
    ref = oracle.qmatmul(lay.packed, lay.scales_raw, lay.biases_raw, synth.BF16, xv, K, 4, 64)
    assert oracle.max_rel_err(outs[0], ref) < 1e-3
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
    assert np.array_equal(outs[0].view(np.uint32), outs[2].view(np.uint32))


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_full_precision_gemm_at_its_edges(mlxq, oracle, bits):
    # the GEMM behind batches whose operands may not be rounded to fp16: one step of K and more, all group sizes, one to
    # several row tiles and tokens tiles of 32 / 64 / 128, K split over CTAs (K = 2048: four segments) and not, a row
    # bias, strided rows with NaN padding.  The bound: an activation is kept to 2^-22 (two fp16 numbers), each of up to eight
    # tensor-core steps of a group drops what lies below 2^-25 of its sum, the rest is fp32: 2^-22 + 8 * 2^-25 < 5e-7 of
    # the terms, which cancel by less than two -- 1e-6 normwise.
    for gs, x_dtype, T, O, K in [(32, 0, 17, 41, 128), (64, 0, 33, 129, 2048), (128, 0, 129, 264, 1280), (64, 1, 64, 127, 640),
                                 (32, 2, 65, 300, 1152), (128, 2, 32, 40, 2048)]:
        if bits == 4 and x_dtype != 0 and K >= 1024:
            x_dtype = 0                                            # (4-bit layers round 16-bit activations' weights to fp16 there)
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, with_bias=True, seed=T + O + bits)
        layer = DevLayer.from_fixture(mlxq, fx)
        x = oracle.RNG(T + K).floats(T * K).reshape(T, K)
        xr = as_dtype(x, x_dtype).float().cpu().numpy()
        got = run(layer, x, T, x_dtype=x_dtype, x_stride=K + 8, y_stride=O + 3)
        mlxq.streamStatus(None, 0)
        if bits == 4 and x_dtype != 0:
            bar = 5e-4                                             # K = 640: the fp16-weight GEMM's bar
        else:
            bar = 1e-6
        ref = _ref(oracle, fx, xr, K, bits, gs, oracle.BF16, bias=fx.bias)
        nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
        assert nrm < bar, f"bits {bits} gs {gs} x dtype {x_dtype} T {T} {O}x{K}: normwise {nrm}"


def test_captured_long_batches_need_no_allocation_nodes(mlxq, oracle):
    # a stream under capture keeps the kernels that use no scratch memory; the results agree within both paths' fp32 sums
    O, K, T = 200, 1024, 40
    fx = oracle.QuantFixture(O=O, K=K, bits=8, gs=64, seed=9)
    layer = DevLayer.from_fixture(mlxq, fx)
    xv = oracle.RNG(3).floats(T * K).reshape(T, K)
    x = torch.from_numpy(xv).cuda()
    y = torch.full((T, O), float("nan"), device="cuda")
    layer.linear.encode(None, x, K, y, O, T)
    torch.cuda.synchronize()
    eager = y.cpu().numpy()
    y.fill_(float("nan"))
    layer.linear.encode(None, x[:16], K, y, O, 16)                 # (function attributes are set outside the capture)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        layer.linear.encode(torch.cuda.current_stream(), x, K, y, O, T)
    g.replay()
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    assert float(np.linalg.norm(y.cpu().numpy() - eager) / np.linalg.norm(eager)) < 5e-6


@pytest.mark.parametrize("bits,gs,K,O", [(8, 64, 12288, 40), (4, 64, 12288, 24), (2, 32, 256, 40), (6, 128, 14336, 24)])
@pytest.mark.parametrize("x_dtype", [0, 2])
def test_full_precision_gemm_at_any_magnitude(mlxq, oracle, bits, gs, K, O, x_dtype):
    # activations outside fp16's range: tokens of 1e-38 ... 1e30, one whose elements span ten orders of magnitude, one of
    # zeros, and next to them one with an infinity.  A token's power of two leaves what lies above 2^-40 of its largest
    # element as exact as at magnitude one, so every token meets the same bar as there (1e-6 of its norm).
    if bits == 4 and x_dtype != 0:
        x_dtype = 0                                                # (16-bit activations on 4-bit layers take the other GEMM)
    fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, seed=bits + K)
    layer = DevLayer.from_fixture(mlxq, fx)
    mags = [1e-38, 1e-20, 1e-5, 1e-4, 1e-3, 1e-2, 1.0, 1e2, 7e4, 1e5, 1e10, 1e30]
    T = len(mags) + 8
    x = oracle.RNG(K + bits).floats(T * K).reshape(T, K)
    for t, m in enumerate(mags):
        x[t] = (x[t].astype(np.float64) * m).astype(np.float32)
    n = len(mags)
    x[n] = (x[n] * np.exp(np.linspace(0.0, 23.0, K))).astype(np.float32)
    x[n + 1] = 0.0
    x[n + 2, 5] = np.inf
    xr = as_dtype(x, x_dtype).float().cpu().numpy()
    got = run(layer, x, T, x_dtype=x_dtype).astype(np.float64)
    mlxq.streamStatus(None, 0)
    finite = [t for t in range(T) if t != n + 2]
    w = np.repeat(oracle.to_float(fx.scales_raw, oracle.BF16), gs, axis=1).astype(np.float64) * fx.q + \
        np.repeat(oracle.to_float(fx.biases_raw, oracle.BF16), gs, axis=1).astype(np.float64)
    ref = xr[finite].astype(np.float64) @ w.T
    for i, t in enumerate(finite):
        if t == n + 1:
            assert not got[t].any()
            continue
        err = float(np.linalg.norm(got[t] - ref[i]) / np.linalg.norm(ref[i]))
        assert err < 1e-6, f"bits {bits} x dtype {x_dtype} token {t} (largest {np.abs(xr[t]).max():.3g}): {err}"
    assert not np.isfinite(got[n + 2]).any()


@pytest.mark.parametrize("gs", [32, 64])
def test_full_precision_gemm_on_long_8_bit_rows(mlxq, oracle, gs):
    # rows beyond 8192 codes on a layer with a row tile for every SM, where K would otherwise be one sum of 132 (264) steps.
    # Rounding 24 times a running sum that grows like their square root: 2^-24 * sqrt(24 / 2) / sqrt(3) = 1.2e-7 of the result;
    # the tensor core drops up to 2^-25 of a group's sum at each of its four steps, half of it on average: 0.6e-7.
    # Together 1.4e-7; one sum gives 2.0e-7 and 2.9e-7.
    O, K, T = 18944, 8448, 20
    rng = np.random.default_rng(gs)
    q = rng.integers(0, 256, (O, K), dtype=np.uint8)
    s = torch.from_numpy((np.abs(rng.standard_normal((O, K // gs))) * 0.002 + 1e-4).astype(np.float32)).to(torch.bfloat16)
    b = (-128.0 * s.float()).to(torch.bfloat16)
    x = torch.from_numpy(rng.standard_normal((T, K)).astype(np.float32)).to(torch.bfloat16)
    lin = mlxq.Linear(torch.from_numpy(q.view(np.int32)).cuda(), s.cuda(), b.cuda(), None, inDim=K)
    y = torch.full((T, O), float("nan"), device="cuda")
    lin.encode(None, x.cuda(), K, y, O, T)
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    rows = rng.choice(O, 96, replace=False)
    w = np.repeat(s.double().numpy()[rows], gs, axis=1) * q[rows] + np.repeat(b.double().numpy()[rows], gs, axis=1)
    ref = x.double().numpy() @ w.T
    nrm = float(np.linalg.norm(y.cpu().numpy()[:, rows] - ref) / np.linalg.norm(ref))
    assert nrm < 1.4e-7, f"gs {gs}: normwise {nrm}"


@pytest.mark.parametrize("bits,x_dtype", [(4, 2), (8, 2), (4, 0)])
def test_gemm_reads_weights_written_just_ahead_in_the_stream(mlxq, bits, x_dtype):
    # A kernel of the library that lets its successor start early (the activation product) writes the packed weights; the
    # GEMM behind it must see all of them.  (Its pre-pass is a dependent launch too, so nothing but its own order of wait and
    # trigger keeps the GEMM from reading ahead.)
    O, K, T = 4096, 4096, 64
    words = O * K * bits // 32
    cols, rows = 4096, words // 4096
    gen = torch.Generator(device="cuda")
    gen.manual_seed(bits)
    w = torch.zeros(words, device="cuda")
    gu = torch.randn((rows, 2 * cols), device="cuda", generator=gen)
    s = (torch.rand((O, K // 64), device="cuda", generator=gen) * 0.01).to(torch.bfloat16)
    lin = mlxq.Linear(w.view(torch.int32).view(O, -1), s, s.clone(), None, inDim=K)
    lin.prepare()
    x = torch.randn((T, K), device="cuda", generator=gen).to({0: torch.float32, 2: torch.bfloat16}[x_dtype])
    y, ref = torch.zeros((T, O), device="cuda"), torch.zeros((T, O), device="cuda")
    mlxq.actMul(None, gu, 2 * cols, cols, rows, mlxq.ACT_SILU, w)
    torch.cuda.synchronize()
    lin.encode(None, x, K, ref, O, T)
    for _ in range(20):
        w.zero_()
        torch.cuda.synchronize()
        mlxq.actMul(None, gu, 2 * cols, cols, rows, mlxq.ACT_SILU, w)
        lin.encode(None, x, K, y, O, T)
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
    mlxq.streamStatus(None, 0)


_ORDINARY_LAUNCHES = """
import importlib, sys, torch
mlxq, out = importlib.import_module("mlx-runner_b200"), {}
gen = torch.Generator(device="cuda"); gen.manual_seed(3)
for bits in (4, 8):
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (264, 512 * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = torch.rand((264, 8), device="cuda", generator=gen).to(torch.bfloat16)
    lin = mlxq.Linear(w, s, s.clone(), None, inDim=512)
    for T in (1, 3, 20, 200):
        x = torch.randn((T, 512), device="cuda", generator=gen).to(torch.bfloat16)
        y = torch.zeros((T, 264), device="cuda")
        lin.encode(None, x, 512, y, 264, T)
        a = torch.zeros((T, 132), device="cuda")
        mlxq.actMul(None, y, 264, 132, T, mlxq.ACT_SILU, a)
        out[bits, T] = (y.cpu(), a.cpu())
torch.save(out, sys.argv[1])
"""


def test_ordinary_launches_give_the_same_bits(mlxq, tmp_path):
    # MLXQ_PDL=0 (read once per process, hence the child processes) turns every dependent launch into an ordinary one
    import os
    import subprocess
    import sys
    got = []
    for v in ("0", "1"):
        out = tmp_path / f"pdl{v}.pt"
        subprocess.run([sys.executable, "-c", _ORDINARY_LAUNCHES, str(out)], check=True, timeout=300, env={**os.environ, "MLXQ_PDL": v},
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
        got.append(torch.load(out))
    for key, (y, a) in got[0].items():
        assert torch.equal(y, got[1][key][0]) and torch.equal(a, got[1][key][1]), key


def _sampled(oracle, fx, xr, rows, tokens):
    """The oracle's outputs of some rows for some tokens."""
    return oracle.qmatmul(fx.packed[rows], fx.scales_raw[rows], fx.biases_raw[rows], oracle.BF16, np.ascontiguousarray(xr[tokens]), fx.K, fx.bits, fx.gs)


@pytest.mark.parametrize("bits", [2, 5, 8])
def test_full_precision_gemm_in_eight_segments(mlxq, oracle, bits):
    # 4096 codes on three row tiles: K over eight CTAs
    O, K, T = 300, 4096, 70
    fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=64, scale_type=oracle.BF16, seed=bits)
    layer = DevLayer.from_fixture(mlxq, fx)
    for x_dtype in (0, 2):
        x = oracle.RNG(T).floats(T * K).reshape(T, K)
        xr = as_dtype(x, x_dtype).float().cpu().numpy()
        got = run(layer, x, T, x_dtype=x_dtype, y_stride=O + 3)
        ref = _ref(oracle, fx, xr, K, bits, 64, oracle.BF16)
        assert float(np.linalg.norm(got - ref) / np.linalg.norm(ref)) < 1e-6
    mlxq.streamStatus(None, 0)


@pytest.mark.parametrize("K", [128, 256, 384])
def test_full_precision_gemm_on_short_4_bit_rows(mlxq, oracle, K):
    # 4-bit layers with 16-bit activations take it below 512 codes (one fp16 part, codes in the permuted order)
    O, T = 264, 90
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, scale_type=oracle.BF16, with_bias=True, seed=K)
    layer = DevLayer.from_fixture(mlxq, fx)
    for x_dtype in (1, 2):
        x = oracle.RNG(T + K).floats(T * K).reshape(T, K)
        xr = as_dtype(x, x_dtype).float().cpu().numpy()
        got = run(layer, x, T, x_dtype=x_dtype, x_stride=K + 8)
        ref = _ref(oracle, fx, xr, K, 4, 64, oracle.BF16, bias=fx.bias)
        assert float(np.linalg.norm(got - ref) / np.linalg.norm(ref)) < 1e-6
    mlxq.streamStatus(None, 0)


def test_full_precision_gemm_in_slices_of_tokens(mlxq, oracle):
    # 12288 fp32 codes a token on five row tiles: a slice holds 1408 tokens (scratch for both parts and eight sums an output), so 4500 tokens
    # take several turns over the same scratch memory, the last one shorter.  Tokens on both sides of every multiple of 128 that may
    # be a boundary against the oracle, and every token against the same one in a short batch, bit for bit.
    O, K, T = 520, 12288, 4500
    fx = oracle.QuantFixture(O=O, K=K, bits=8, gs=64, scale_type=oracle.BF16, seed=3)
    layer = DevLayer.from_fixture(mlxq, fx)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    x = torch.rand((T, K), device="cuda", generator=gen) * 2 - 1
    y, part = torch.full((T, O), float("nan"), device="cuda"), torch.full((T, O), float("nan"), device="cuda")
    layer.linear.encode(None, x, K, y, O, T)
    for t0 in range(0, T, 100):
        layer.linear.encode(None, x[t0:], K, part[t0:], O, min(100, T - t0))
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    assert torch.equal(y, part)
    tokens = [t for b in range(0, T, 128) for t in (b - 1, b) if 0 <= t < T] + [T - 1]
    ref = _ref(oracle, fx, x[tokens].cpu().numpy(), K, 8, 64, oracle.BF16)
    assert float(np.linalg.norm(y[tokens].cpu().numpy() - ref) / np.linalg.norm(ref)) < 1e-6


@pytest.mark.parametrize("T", [17, 77, 128])
def test_tall_tile_of_short_batches_on_many_rows(mlxq, oracle, T):
    # more row tiles than one round of the SMs holds, at most 128 tokens: 256 rows a tile, the last one ragged.  The same tokens
    # in a batch of 256 take the wide tile: the sums are the same, bit for bit.
    O, K = 19001, 512
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, scale_type=oracle.BF16, with_bias=True, seed=T)
    layer = DevLayer.from_fixture(mlxq, fx)
    assert layer.linear.gemmTileTokens(T) == 128
    x = oracle.RNG(T).floats(256 * K).reshape(256, K)
    xr = as_dtype(x, 2).float().cpu().numpy()
    got, wide = run(layer, x[:T], T, x_dtype=2, y_stride=O + 3), run(layer, x, 256, x_dtype=2)
    mlxq.streamStatus(None, 0)
    assert np.array_equal(got.view(np.uint32), wide[:T].view(np.uint32))
    rows = np.r_[0:130, 9000:9300, 18900:O]
    ref = _sampled(oracle, fx, xr, rows, np.arange(T)) + fx.bias[rows]
    assert float(np.linalg.norm(got[:, rows] - ref) / np.linalg.norm(ref)) < 5e-4
