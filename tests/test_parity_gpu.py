"""GPU parity tests: the CUDA layer, called through the C ABI, against the CPU oracle on the same seeded
inputs.  The matrix mirrors the reference's kernel tests (Tests/MLXEngineTests/KernelTests.swift:126-297):
same shapes, same xorshift seeds, same error metric (max |got-ref| / max(1,|ref|)).

Tolerance: 1e-3 (the bar this build states; the reference's own bar is 2e-3), 5e-3 for the gated output
(as KernelTests.swift:211) and 1e-5 for the dequantising lookup (KernelTests.swift:295).  Unpacked codes
must be bit-exact."""
import importlib

import numpy as np
import pytest
import torch

from helpers import TORCH_DT, DevLayer, as_dtype, dev, run

synth = importlib.import_module("mlx-runner_b200.synth")

pytestmark = pytest.mark.gpu

TOL = 1e-3


def on_kernel(monkeypatch, name):
    """MLXQ_DECODE (read at every call): the small-batch kernel to take, or the dispatch's own choice."""
    if name is None:
        monkeypatch.delenv("MLXQ_DECODE", raising=False)
    else:
        monkeypatch.setenv("MLXQ_DECODE", name)


def close(oracle, got, ref, label, tol=TOL):
    err = oracle.max_rel_err(got, ref)
    assert err < tol, f"{label}: max relative error {err}"


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_quantized_matches_reference(mlxq, oracle, bits):
    # KernelTests.swift:128-146
    K, O = 512, 40
    for gs in (32, 64, 128):
        for st in (oracle.F16, oracle.BF16):
            fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=st)
            layer = DevLayer.from_fixture(mlxq, fx)
            for T in (1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 33):
                x = oracle.RNG(T * 31 + bits).floats(T * K).reshape(T, K)
                close(oracle, run(layer, x, T), fx.reference(x), f"bits {bits} gs {gs} st {st} T {T}")


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_unpacked_codes_are_bit_exact(mlxq, oracle, bits):
    fx = oracle.QuantFixture(O=37, K=544, bits=bits, gs=32, seed=bits + 100)
    layer = DevLayer.from_fixture(mlxq, fx)
    out = torch.zeros((37, 544), dtype=torch.uint8, device="cuda")
    layer.linear.unpackCodes(None, out)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got, fx.q)
    assert np.array_equal(got, oracle.unpack(fx.packed, 544, bits))


@pytest.mark.parametrize("bits", [3, 4, 8])
def test_prefill_tiles_match_reference(mlxq, oracle, bits):
    # KernelTests.swift:150-164: long batches, odd O, K % 64 != 0
    for T, O, K in [(64, 41, 1056), (128, 41, 544), (517, 41, 544), (96, 2050, 544), (128, 2050, 544), (517, 520, 544)]:
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=32, seed=T + O)
        layer = DevLayer.from_fixture(mlxq, fx)
        x = oracle.RNG(T * 7 + bits).floats(T * K).reshape(T, K)
        ref = oracle.qmatmul(fx.packed, fx.scales_raw, fx.biases_raw, fx.scale_type, x, K, bits, 32)
        close(oracle, run(layer, x, T), ref, f"bits {bits} T {T} O {O} K {K}")


def test_batches_agree_bitwise(mlxq, oracle):
    # KernelTests.swift:168-184: a token's output does not depend on the batch it was computed in
    # (checked within each kernel family: the matvec up to 16 tokens, the GEMM above).
    O, K = 2050, 1024
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, seed=3)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = oracle.RNG(11).floats(256 * K).reshape(256, K)
    full16 = run(layer, x[:16], 16).view(np.uint32)
    for T in (9, 12):
        assert np.array_equal(run(layer, x[:T], T).view(np.uint32), full16[:T]), f"T {T} vs T 16"
    # and a decode call is reproducible bit for bit (sums are formed in a fixed order)
    assert np.array_equal(run(layer, x[:1], 1).view(np.uint32), run(layer, x[:1], 1).view(np.uint32))
    full = run(layer, x, 256).view(np.uint32)
    for T in (33, 96, 131):
        assert np.array_equal(run(layer, x[:T], T).view(np.uint32), full[:T]), f"T {T} vs T 256"


@pytest.mark.parametrize("K", [1152, 1536, 2304, 2560, 896, 1664, 6912])
def test_four_bit_decode_with_partial_pass(mlxq, oracle, K):
    # KernelTests.swift:188-199
    O = 24
    for gs in (32, 64, 128):
        if K % gs:
            continue
        fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=gs, seed=K)
        layer = DevLayer.from_fixture(mlxq, fx)
        x = oracle.RNG(K).floats(K).reshape(1, K)
        close(oracle, run(layer, x, 1), fx.reference(x), f"K {K} gs {gs}")


def test_gated_output_matches_reference(mlxq, oracle):
    # KernelTests.swift:202-212: y = act(x . W^T) * e, tanh-GELU, e read at an offset
    O, K = 40, 1536
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, seed=21)
    layer = DevLayer.from_fixture(mlxq, fx)
    rng = oracle.RNG(6)
    x = rng.floats(K) * np.float32(4)
    e = rng.floats(2 * O)
    xd, ed = as_dtype(x, 0), as_dtype(e, 0)
    for act in (0, 1, 2):
        yd = torch.zeros(O, dtype=torch.float32, device="cuda")
        layer.linear.encodeGated(None, xd, yd, ed[O:], act)
        torch.cuda.synchronize()
        g = fx.reference(x.reshape(1, K))[0]
        if act == 1:
            ref = 0.5 * g * (1 + np.tanh(np.float32(0.7978845608) * (g + np.float32(0.044715) * g * g * g))) * e[O:]
            close(oracle, yd.cpu().numpy(), ref.astype(np.float32), "gated output (formula of the reference test)", 5e-3)
        close(oracle, yd.cpu().numpy(), oracle.act_mul(act, g, e[O:]), f"gated output act {act}", 5e-3)


def _fused_parts(mlxq, oracle, K):
    fxs = [oracle.QuantFixture(O=o, K=K, bits=4, gs=64, with_bias=True, seed=s) for o, s in [(64, 1), (16, 2), (16, 3)]]
    return fxs, [DevLayer.from_fixture(mlxq, f, name=f"p{i}") for i, f in enumerate(fxs)]


def test_fused_decode_with_bias_matches_separate(mlxq, oracle):
    # KernelTests.swift:214-227
    K = 256
    fxs, layers = _fused_parts(mlxq, oracle, K)
    lins = [l.linear for l in layers]
    assert mlxq.Linear.fusable(lins)
    x = oracle.RNG(99).floats(K)
    yd = torch.zeros(96, dtype=torch.float32, device="cuda")
    mlxq.Linear.encodeFusedDecode(None, lins, as_dtype(x, 0), yd)
    torch.cuda.synchronize()
    ref = np.concatenate([f.reference(x.reshape(1, K))[0] for f in fxs])
    close(oracle, yd.cpu().numpy(), ref, "fused q/k/v")


@pytest.mark.parametrize("K", [512, 1152, 544, 1056])
def test_small_batch_four_bit_matches_reference(mlxq, oracle, K):
    # KernelTests.swift:232-252: strided x / y, NaN padding that must not be read, rows that end inside a warp
    for O, gs in [(40, 64), (44, 32), (40, 128)]:
        if K % gs:
            continue
        for st in (oracle.F16, oracle.BF16):
            fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=gs, scale_type=st, seed=K + O)
            layer = DevLayer.from_fixture(mlxq, fx)
            for T in (2, 3, 4, 5, 8):
                assert mlxq.Linear.canFuse([layer.linear], T)
                x = oracle.RNG(T * 131 + K).floats(T * K).reshape(T, K)
                got = run(layer, x, T, x_stride=K + 4, y_stride=O + 3)
                close(oracle, got, fx.reference(x), f"K {K} O {O} gs {gs} st {st} T {T}")


def test_small_batch_fused_with_bias_matches_separate(mlxq, oracle):
    # KernelTests.swift:255-269
    K = 1152
    fxs, layers = _fused_parts(mlxq, oracle, K)
    lins = [l.linear for l in layers]
    for T in (2, 7, 8):
        x = oracle.RNG(T).floats(T * K).reshape(T, K)
        yd = torch.zeros((T, 96), dtype=torch.float32, device="cuda")
        mlxq.Linear.encodeFusedDecode(None, lins, as_dtype(x, 0), yd, xStride=K, yStride=96, T=T)
        torch.cuda.synchronize()
        ref = np.concatenate([f.reference(x) for f in fxs], axis=1)
        close(oracle, yd.cpu().numpy(), ref, f"fused q/k/v T {T}")


@pytest.mark.parametrize("kernel", [None, "tok", "tc"])
@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_small_batches_every_width_and_group(mlxq, oracle, monkeypatch, bits, kernel):
    # Two to sixteen tokens take one of the two decode kernels whose accumulator columns are tokens (where they serve the width
    # and group size; the others fall to the general kernels): both 16-bit scale types, fp16 and fp32 activations, a row
    # count that ends inside a block, group counts that leave windows of eight groups partly empty.  The bar is the
    # fp32 reassociation noise of a K-long sum, far below the 1e-3 of the reference's own tests.
    on_kernel(monkeypatch, kernel)
    K, O = 1536, 72
    for gs in (32, 64, 128):
        for st in (oracle.F16, oracle.BF16):
            fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=st, with_bias=(gs == 64), seed=bits * 7 + gs)
            layer = DevLayer.from_fixture(mlxq, fx)
            for T, x_dtype in ((2, 1), (5, 1), (8, 1), (9, 1), (16, 1), (3, 0), (8, 0), (4, 2)):
                x = oracle.RNG(T * 17 + gs + bits).floats(T * K).reshape(T, K)
                xr = as_dtype(x, x_dtype).float().cpu().numpy()
                got = run(layer, x, T, x_dtype=x_dtype, x_stride=K + 8, y_stride=O + 5)
                # (fp32 activations ride as two fp16 columns: the split leaves 2^-22 of every product)
                close(oracle, got, fx.reference(xr), f"bits {bits} gs {gs} st {st} T {T} x {x_dtype}", 1e-4 if x_dtype == 0 else 3e-5)


@pytest.mark.parametrize("kernel", ["tok", "tc"])
@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_small_batches_of_long_rows(mlxq, oracle, monkeypatch, bits, kernel):
    # rows of 6144 codes and more: single CTAs, and clusters where those do not hold the tokens -- even and uneven slices, fewer
    # blocks than clusters and several rounds of them, 16 tokens of 16-bit activations (a wider cluster where the slices do not
    # fit)
    on_kernel(monkeypatch, kernel)
    for gs, K, O, T, x_dtype in ((64, 6144, 41, 2, 0), (32, 6656, 600, 6, 0), (128, 12288, 24, 8, 0), (64, 14336, 40, 16, 1), (64, 6400, 700, 5, 2),
                                (64, 6144, 700, 8, 0), (64, 12288, 600, 6, 0), (64, 6144, 41, 16, 1), (128, 14336, 600, 10, 2)):
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, with_bias=(gs == 64), seed=bits + K)
        layer = DevLayer.from_fixture(mlxq, fx)
        x = oracle.RNG(T + K + bits).floats(T * K).reshape(T, K)
        xr = as_dtype(x, x_dtype).float().cpu().numpy()
        got = run(layer, x, T, x_dtype=x_dtype, x_stride=K + 8, y_stride=O + 5)
        mlxq.streamStatus(None, 0)
        # The bar of the small batches above holds for 1536 terms and is in units of max(1, |reference|): the rounding noise of
        # a sum of K such terms is sqrt(K / 1536) times that.
        close(oracle, got, fx.reference(xr), f"bits {bits} gs {gs} {O}x{K} T {T} x {x_dtype}", (1e-4 if x_dtype == 0 else 3e-5) * (K / 1536) ** 0.5)


@pytest.mark.parametrize("T,O", [(5, 17), (5, 16 * 37 * 3), (7, 16 * 75), (5, 40)])
def test_cluster_kernel_with_half_warps_at_different_turns(mlxq, oracle, monkeypatch, T, O):
    # odd tokens times odd blocks a cluster: the last rounds of the loops before the cluster's barriers, and of the block
    # ends, are run by half a warp.  One call after the other on the same buffers, so that a CTA that left early would
    # read the next call's sums.
    on_kernel(monkeypatch, "tok")
    K, gs = 12288, 64
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=gs, scale_type=oracle.BF16, seed=O)
    layer = DevLayer.from_fixture(mlxq, fx)
    x_dtype = 0 if T == 5 else 1
    xv = oracle.RNG(T + O).floats(T * K).reshape(T, K)
    xd = as_dtype(xv, x_dtype)
    y = torch.full((T, O), float("nan"), device="cuda")
    for _ in range(3):
        layer.linear.encode(None, xd, K, y, O, T)
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    close(oracle, y.cpu().numpy(), fx.reference(xd.float().cpu().numpy()), f"{O}x{K} T {T}", (1e-4 if x_dtype == 0 else 3e-5) * (K / 1536) ** 0.5)


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("x_dtype,T", [(0, 7), (0, 8), (1, 12), (2, 13)])
@pytest.mark.parametrize("kernel", ["tok", "tc"])
def test_cluster_kernel_at_any_magnitude(mlxq, oracle, monkeypatch, bits, x_dtype, T, kernel):
    # batches that the clusters (and the tensor-memory kernel) serve in the place of kernels that multiply in fp32: tokens of 1e-30 ... 1e30 side by side, one
    # of zeros, one whose elements span ten orders of magnitude; in fp16 down to its subnormal numbers.  A token's power of two
    # leaves what lies above 2^-40 of its largest element as exact as at magnitude one; the bar there is that of the sums: the
    # uncentred codes' are up to four times the result's at 2 bits, 14336 terms in 16 slices, 2^-24 * sqrt(14336 / 16 / 8) * 4
    # and the bias term's as much again: 5e-6.
    if bits == 8 and x_dtype != 0:
        T = 8                                                      # (8 bits, 16-bit activations: two half batches, no cluster beyond)
    on_kernel(monkeypatch, kernel)
    K, gs = 14336, 64
    for O in (40, 16 * 37 + 1):
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, seed=bits + O)
        layer = DevLayer.from_fixture(mlxq, fx)
        x = oracle.RNG(T + bits).floats(T * K).reshape(T, K)
        mags = [1.0] * 3 if bits == 8 and x_dtype != 0 else [1e-6, 1e-3, 3e4] if x_dtype == 1 else [1e-30, 1e-5, 1e30]
        for t, m in enumerate(mags):
            x[t] = x[t] * np.float32(m)
        x[3] = 0.0
        if x_dtype != 1 and bits != 8:
            x[4] = x[4] * np.exp(np.linspace(0.0, 23.0, K)).astype(np.float32)
        xd = as_dtype(x, x_dtype)
        y = torch.full((T, O + 3), float("nan"), device="cuda")
        layer.linear.encode(None, xd, K, y, O + 3, T)
        torch.cuda.synchronize()
        mlxq.streamStatus(None, 0)
        got = y.cpu().numpy()[:, :O].astype(np.float64)
        w = np.repeat(oracle.to_float(fx.scales_raw, oracle.BF16), gs, axis=1).astype(np.float64) * fx.q + \
            np.repeat(oracle.to_float(fx.biases_raw, oracle.BF16), gs, axis=1).astype(np.float64)
        ref = xd.double().cpu().numpy() @ w.T
        for t in range(T):
            if t == 3:
                assert not got[t].any()
                continue
            err = float(np.linalg.norm(got[t] - ref[t]) / np.linalg.norm(ref[t]))
            assert err < 5e-6, f"bits {bits} x dtype {x_dtype} {O}x{K} token {t} of {T}: {err}"


@pytest.mark.parametrize("x_dtype,T", [(0, 9), (0, 16), (2, 16), (0, 24), (2, 24)])
@pytest.mark.parametrize("kernel", [None, "tok"])
def test_batches_beyond_the_persistent_kernels_keep_fp32_products(mlxq, oracle, monkeypatch, x_dtype, T, kernel):
    # calls that no persistent kernel holds on single CTAs, as one call or as two halves, multiply in fp32, or on the
    # tensor-memory kernel in scaled fp16 parts: activations of 1e5, which an fp16 operand cannot hold unscaled, and of 1e-5,
    # which it holds to a few bits.  24 tokens: the paths without
    # scratch memory (static, captured, three layers in one launch).  The bar: fp32 sums of 14336 terms in 32 lanes, each
    # rounding 448 times (2^-24 * sqrt(448 / 3) = 7e-7 of the result; measured 3e-7).
    on_kernel(monkeypatch, kernel)
    K, O, bits, gs = 14336, 24, 8, 64
    fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, seed=T)
    layer = DevLayer.from_fixture(mlxq, fx)
    for mag in (1e5, 1e-5):
        x = oracle.RNG(T).floats(T * K).reshape(T, K) * np.float32(mag)
        xd = as_dtype(x, x_dtype)
        ref = oracle.qmatmul(fx.packed, fx.scales_raw, fx.biases_raw, oracle.BF16, xd.float().cpu().numpy(), K, bits, gs)

        def check(y, what):
            torch.cuda.synchronize()
            got = y.cpu().numpy()[:, :O]
            nrm = float(np.linalg.norm(got - ref) / np.linalg.norm(ref))
            assert nrm < 7e-7, f"{what}, x dtype {x_dtype}, {T} tokens of {mag:g}: {nrm}"

        y = torch.full((T, O), float("nan"), device="cuda")
        if T <= 16:
            layer.linear.encode(None, xd, K, y, O, T)
            check(y, "forward")
            continue
        layer.linear.encodeStatic(None, xd, K, y, O, T)
        check(y, "static")
        y.fill_(float("nan"))
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            layer.linear.encode(torch.cuda.current_stream(), xd, K, y, O, T)
        g.replay()
        check(y, "captured")
        y3 = torch.full((T, 3 * O), float("nan"), device="cuda")
        mlxq.Linear.encodeFusedDecode(None, [layer.linear] * 3, xd, y3, xStride=K, yStride=3 * O, T=T)
        check(y3, "fused")


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_one_fp32_token_every_width_and_group(mlxq, oracle, bits):
    # one fp32 token: its two fp16 parts on the kernel compiled for the group size, where slices of K hold whole drain
    # cycles of four groups, and on the general plan where they do not (K = 768); odd numbers of blocks and of steps
    for gs in (32, 64, 128):
        for K, O in ((768, 24), (1024, 40), (1536, 72), (5120, 17)):
            fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16 if K % 1024 else oracle.F16, with_bias=(O == 72), seed=bits + gs + K)
            layer = DevLayer.from_fixture(mlxq, fx)
            x = oracle.RNG(K + gs + bits).floats(K).reshape(1, K)
            # (the split leaves 2^-22 of every product, the sums are fp32: the small batches' bar for fp32 activations)
            close(oracle, run(layer, x, 1), fx.reference(x), f"bits {bits} gs {gs} {O}x{K}", 1e-4)


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_quantized_embedding_lookup(mlxq, oracle, bits):
    # KernelTests.swift:287-296 (4-bit there; every width here)
    K, V = 128, 16
    fx = oracle.QuantFixture(O=V, K=K, bits=bits, gs=64)
    layer = DevLayer.from_fixture(mlxq, fx)
    ids = torch.tensor([3, 0, 15, 7], dtype=torch.int32, device="cuda")
    out = torch.zeros((4, K), dtype=torch.float32, device="cuda")
    layer.linear.encodeLookup(None, ids, out, 4)
    mlxq.streamStatus(None, 0)
    ref = fx.dense[[3, 0, 15, 7]]
    close(oracle, out.cpu().numpy(), ref, "embedding", 1e-5)
    assert np.array_equal(out.cpu().numpy(), ref)          # two roundings, as the CPU code evaluates it


def test_lookup_rejects_ids_outside_the_table(mlxq, oracle):
    fx = oracle.QuantFixture(O=16, K=128, bits=4, gs=64)
    layer = DevLayer.from_fixture(mlxq, fx)
    ids = torch.tensor([3, 16, -1, 7], dtype=torch.int32, device="cuda")
    out = torch.full((4, 128), 5.0, dtype=torch.float32, device="cuda")
    layer.linear.encodeLookup(None, ids, out, 4)
    with pytest.raises(mlxq.GPUFailure, match="lookup id"):
        mlxq.streamStatus(None, 0)
    o = out.cpu().numpy()
    assert np.all(o[1] == 0) and np.all(o[2] == 0) and np.array_equal(o[0], fx.dense[3])
    mlxq.streamStatus(None, 0)                              # the error word is cleared after it is reported


def test_row_list_matvec(mlxq, oracle):
    # head_exact, Kernels.swift:2752-2787: only the listed rows are written
    O, K = 300, 512
    fx = oracle.QuantFixture(O=O, K=K, bits=6, gs=64, seed=5)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = oracle.RNG(8).floats(K)
    rows = [5, 299, 0, 17, -3, 300, 123]
    lst = torch.tensor(rows + [1, 2], dtype=torch.int32, device="cuda")
    cnt = torch.tensor([len(rows)], dtype=torch.int32, device="cuda")
    y = torch.full((O,), -7.0, dtype=torch.float32, device="cuda")
    layer.linear.encodeRows(None, as_dtype(x, 0), y, cnt, lst, len(rows) + 2)
    torch.cuda.synchronize()
    got, ref = y.cpu().numpy(), fx.reference(x.reshape(1, K))[0]
    valid = [r for r in rows if 0 <= r < O]
    close(oracle, got[valid], ref[valid], "row list")
    untouched = np.ones(O, dtype=bool)
    untouched[valid] = False
    assert np.all(got[untouched] == -7.0)


@pytest.mark.parametrize("x_dtype,y_dtype", [(1, 0), (2, 0), (1, 1), (2, 2), (0, 2)])
def test_activation_and_output_dtypes(mlxq, oracle, x_dtype, y_dtype):
    # the benchmark configurations feed f16 / bf16 activations; outputs may be 16-bit too
    O, K = 72, 1024
    for bits in (4, 6):
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=64, with_bias=True, seed=bits)
        layer = DevLayer.from_fixture(mlxq, fx)
        for T in (1, 4, 7):
            x = oracle.RNG(T + 50).floats(T * K).reshape(T, K)
            xr = as_dtype(x, x_dtype).float().cpu().numpy()            # what the kernel actually sees
            ref = fx.reference(xr)
            got = run(layer, x, T, x_dtype=x_dtype, y_dtype=y_dtype)
            tol = TOL if y_dtype == 0 else (2e-3 if y_dtype == 1 else 1e-2)   # output rounding: f16 2^-11, bf16 2^-8
            close(oracle, got, ref, f"bits {bits} x {x_dtype} y {y_dtype} T {T}", tol)


def test_unaligned_rows_and_odd_groups(mlxq, oracle):
    # rows that are not 16-byte multiples (K*bits/8 % 16 != 0) and group sizes that are only multiples of 8
    for bits, K, gs in [(3, 64, 8), (5, 96, 24), (6, 80, 8), (4, 72, 24), (2, 208, 16), (8, 24, 8), (4, 40, 40)]:
        fx = oracle.QuantFixture(O=19, K=K, bits=bits, gs=gs, seed=K)
        layer = DevLayer.from_fixture(mlxq, fx)
        for T in (1, 3):
            x = oracle.RNG(K + T).floats(T * K).reshape(T, K)
            close(oracle, run(layer, x, T, x_stride=K + (4 - K % 4) % 4 + 4), fx.reference(x), f"bits {bits} K {K} gs {gs} T {T}")


def test_misaligned_x_is_rejected(mlxq, oracle):
    fx = oracle.QuantFixture(O=8, K=64, bits=4, gs=32)
    layer = DevLayer.from_fixture(mlxq, fx)
    xb = torch.zeros(2 * 70, dtype=torch.float32, device="cuda")
    yb = torch.zeros(2 * 8, dtype=torch.float32, device="cuda")
    with pytest.raises(mlxq.InvalidArgument, match="16-byte"):
        layer.linear.encode(None, xb[1:], 64, yb, 8, 1)
    with pytest.raises(mlxq.InvalidArgument, match="16-byte"):
        layer.linear.encode(None, xb, 66, yb, 8, 2)
    with pytest.raises(mlxq.InvalidArgument):
        layer.linear.encode(None, xb, 64, yb, 8, 0)


def test_row_permutation_and_concat(mlxq, oracle):
    # permuteRows / concatRows, Transformer.swift:113-151
    K = 256
    a = oracle.QuantFixture(O=24, K=K, bits=4, gs=64, seed=1)
    b = oracle.QuantFixture(O=16, K=K, bits=4, gs=64, seed=2)
    la, lb = DevLayer.from_fixture(mlxq, a), DevLayer.from_fixture(mlxq, b)
    x = oracle.RNG(4).floats(K).reshape(1, K)
    cat = mlxq.Linear.concatRows(la.linear, lb.linear, "ab")
    assert cat is not None and cat.outDim == 40
    close(oracle, run(cat, x, 1), np.concatenate([a.reference(x), b.reference(x)], axis=1), "concatRows")
    perm = list(np.random.default_rng(0).permutation(24))
    la.linear.permuteRows(perm)
    close(oracle, run(la, x, 1), a.reference(x)[:, perm], "permuteRows")
    with pytest.raises(mlxq.InvalidOutput):
        la.linear.permuteRows([0] * 24)


def test_baseline_shapes_against_oracle(mlxq, oracle):
    # config 1 of the benchmark (4096 x 4096, 4-bit g64, fp32 x) and a slice of the config-2 sweep at full K
    synth = __import__("importlib").import_module("mlx-runner_b200.synth")
    lay = synth.make_layer(4096, 4096, 4, 64, synth.F16, seed=0, bias_noise=True)
    assert np.array_equal(lay.packed.view(np.uint8), oracle.pack_fast(lay.q, 4))
    layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, lay.scale_dtype, 4096)
    _, x = synth.make_activations(1, 4096, synth.F32, seed=1)
    ref = oracle.qmatmul(lay.packed, lay.scales_raw, lay.biases_raw, lay.scale_dtype, x, 4096, 4, 64)
    close(oracle, run(layer, x, 1), ref, "config 1")
    for bits, gs in [(2, 32), (3, 64), (5, 128), (6, 64), (8, 32)]:
        lay = synth.make_layer(688, 4096, bits, gs, synth.F16, seed=bits)
        layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, lay.scale_dtype, 4096)
        for M in (1, 2, 4, 8):
            _, x = synth.make_activations(M, 4096, synth.F16, seed=M)
            ref = oracle.qmatmul(lay.packed, lay.scales_raw, lay.biases_raw, lay.scale_dtype, x, 4096, bits, gs)
            close(oracle, run(layer, x, M, x_dtype=1), ref, f"config 2 bits {bits} gs {gs} M {M}")


def test_committed_golden_cases(mlxq, oracle):
    # every bit width x group size of tests/golden/qlinear_cases.npz: codes bit-exact, outputs within 1e-3
    import golden_cases
    for c in golden_cases.load():
        layer = DevLayer(mlxq, c.packed, c.scales, c.biases, c.sdt, c.K, bias_raw=c.bias, name=c.name)
        codes = torch.full((c.O, c.K), 255, dtype=torch.uint8, device="cuda")
        layer.linear.unpackCodes(None, codes)
        torch.cuda.synchronize()
        assert np.array_equal(codes.cpu().numpy(), c.q), c.name
        for T in (1, c.T):
            got = run(layer, c.x[:T], T)
            assert oracle.max_rel_err(got, c.y[:T]) < 1e-3, f"{c.name} T={T}"
    mlxq.streamStatus(None, 0)


@pytest.mark.parametrize("bits,T,O", [(5, 1, 11008), (4, 8, 11008), (4, 1, 40000), (8, 2, 11008)])
def test_tall_layers_and_larger_batches_run_clean(mlxq, oracle, bits, T, O):
    # benchmark-sized layers whose CTAs hold more 16-row blocks than the shared-memory ring: outputs against the
    # oracle on a sample of rows, and the stream's error word stays clear (a bounded wait that ran out would set it)
    K = 4096
    lay = synth.make_layer(O, K, bits, 64, synth.F16, seed=bits + T, keep_codes=False)
    layer = DevLayer(mlxq, lay.packed, lay.scales_raw, lay.biases_raw, synth.F16, K)
    _, x = synth.make_activations(T, K, synth.F16, seed=3)
    got = run(layer, x, T, x_dtype=1)
    mlxq.streamStatus(None, 0)
    rows = np.sort(np.random.default_rng(O).choice(O, size=96, replace=False))
    ref = oracle.qmatmul(lay.packed[rows], lay.scales_raw[rows], lay.biases_raw[rows], synth.F16, x, K, bits, 64)
    assert oracle.max_rel_err(got[:, rows], ref) < 1e-3


def test_block_maxima_and_greedy_token_are_exact(mlxq, oracle):
    # first pass of the token selection and the greedy pass over it, bit for bit against the oracle: vocabulary-sized
    # rows, a ragged last block, a row stride that breaks 16-byte alignment (scalar path), equal maxima, NaN, -inf
    g = np.random.default_rng(9)
    for V, T, stride in ((151936, 3, 151936), (1000, 4, 1003), (256, 1, 256), (37, 2, 40)):
        x = g.standard_normal((T, stride)).astype(np.float32)
        x[0, V // 3] = x[0, V // 3 + (300 if V > 600 else 1)] = 40.0
        if T > 1:
            x[1, : min(V, 256)] = np.where(np.arange(min(V, 256)) == 1, np.nan, -np.inf)
        ref_m, ref_i = oracle.block_max(x[:, :V], index_base=77)
        nb = ref_m.shape[1]
        xd = torch.from_numpy(x).cuda()
        pairs = torch.zeros((2, T, nb), dtype=torch.int32, device="cuda")
        mlxq.blockMax(None, xd, V, T, stride, pairs, indexBase=77)
        token = torch.zeros(T, dtype=torch.int32, device="cuda")
        value = torch.zeros(T, dtype=torch.float32, device="cuda")
        mlxq.blockArgmax(None, pairs, 1, T, nb, token, value)
        torch.cuda.synchronize()
        got = pairs.cpu().numpy()
        assert np.array_equal(got[0].view(np.float32), ref_m), f"V {V}: block maxima"
        assert np.array_equal(got[1], ref_i), f"V {V}: block indices"
        tok, val = oracle.block_argmax(ref_m, ref_i)
        assert np.array_equal(token.cpu().numpy(), tok) and np.array_equal(value.cpu().numpy(), val), f"V {V}: greedy token"


def test_layers_built_from_safetensors_shards(mlxq, oracle, tmp_path):
    # a model directory written the way MLX writes it (nested names of a multimodal export, 2-byte tensors that leave
    # the following ones off 16-byte boundaries) -> WeightStore on the GPU -> Linear by prefix -> matvec against the oracle
    import json
    import struct
    weights = importlib.import_module("mlx-runner_b200.weights")
    fxs = {"model.layers.0.self_attn.o_proj": oracle.QuantFixture(O=72, K=512, bits=4, gs=64, with_bias=True, seed=3),
           "model.layers.0.mlp.down_proj": oracle.QuantFixture(O=48, K=1024, bits=6, gs=64, scale_type=oracle.BF16, seed=4)}
    header, blobs, off = {}, [], 0

    def put(name, dt, arr):
        nonlocal off
        b = np.ascontiguousarray(arr).tobytes()
        header["language_model." + name] = {"dtype": dt, "shape": list(arr.shape), "data_offsets": [off, off + len(b)]}
        blobs.append(b)
        off += len(b)
    put("model.layer_scalar", "F16", np.array([0.5], dtype=np.float16))                 # shifts everything after it
    for prefix, fx in fxs.items():
        sdt = "F16" if fx.scale_type == oracle.F16 else "BF16"
        put(prefix + ".weight", "U32", fx.packed.view(np.uint32).reshape(fx.O, -1))
        put(prefix + ".scales", sdt, fx.scales_raw)
        put(prefix + ".biases", sdt, fx.biases_raw)
        if fx.bias_raw is not None:
            put(prefix + ".bias", sdt, fx.bias_raw)
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    d = tmp_path / "model"
    d.mkdir()
    with open(d / "model.safetensors", "wb") as fh:
        fh.write(struct.pack("<Q", len(text)) + text + b"".join(blobs))
    store = weights.WeightStore(str(d), device=0)
    assert store.totalBytes == off
    for prefix, fx in fxs.items():
        lin = store.linear(prefix, inDim=fx.K, outDim=fx.O)
        assert (lin.bits, lin.groupSize, lin.outDim) == (fx.bits, fx.gs, fx.O)
        for T in (1, 5):
            x = oracle.RNG(T + fx.O).floats(T * fx.K).reshape(T, fx.K)
            y = torch.zeros((T, fx.O), dtype=torch.float32, device="cuda")
            lin.encode(None, as_dtype(x, 0), fx.K, y, fx.O, T)
            torch.cuda.synchronize()
            close(oracle, y.cpu().numpy(), fx.reference(x), f"{prefix} T {T}")
    with pytest.raises(mlxq.InvalidFile):
        store.linear("model.layers.0.mlp.down_proj", inDim=fxs["model.layers.0.mlp.down_proj"].K, outDim=41)
    # a rank's row shard built from its slice alone (the store stays in host memory, only the slice goes to the GPU)
    host = weights.WeightStore(str(d))
    prefix, fx = "model.layers.0.mlp.down_proj", fxs["model.layers.0.mlp.down_proj"]
    x = oracle.RNG(77).floats(3 * fx.K).reshape(3, fx.K)
    y = torch.zeros((3, fx.O), dtype=torch.float32, device="cuda")
    for r in range(2):
        shard = host.linearShard(prefix, fx.K, r, 2, device=0)
        assert (shard.outDim, shard.totalOut, shard.rowOffset) == (fx.O // 2, fx.O, r * (fx.O // 2))
        shard.encode(None, as_dtype(x, 0), fx.K, y[:, shard.rowOffset:], fx.O, 3)
    torch.cuda.synchronize()
    close(oracle, y.cpu().numpy(), fx.reference(x), "row shards from slices")


def test_gate_up_product_folded_into_the_down_projection(mlxq, oracle):
    # silu_mul / gelu_tanh_mul (Kernels.swift:2004-2030) as a kernel of its own, and folded into the staging of the down
    # projection's activations: both against the oracle's act_mul followed by the layer's reference product
    g = np.random.default_rng(21)
    for bits, K, O in ((4, 1024, 72), (6, 512, 40), (8, 1536, 48)):
        fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=64, seed=bits)
        layer = DevLayer.from_fixture(mlxq, fx)
        for T, act in ((1, 0), (4, 1), (8, 0)):
            stride = 2 * K + 8
            gu = (g.standard_normal((T, stride)) * 1.5).astype(np.float32)
            gud = torch.from_numpy(gu).cuda()
            xref = oracle.act_mul(act, gu[:, :K], gu[:, K:2 * K])
            out = torch.zeros((T, K), dtype=torch.float32, device="cuda")
            mlxq.actMul(None, gud, stride, K, T, act, out)
            y = torch.full((T, O + 3), float("nan"), dtype=torch.float32, device="cuda")
            layer.linear.encodeGLU(None, gud, stride, act, y, O + 3, T)
            torch.cuda.synchronize()
            mlxq.streamStatus(None, 0)
            close(oracle, out.cpu().numpy(), xref, f"act_mul bits {bits} T {T} act {act}", 1e-5)
            close(oracle, y.cpu().numpy()[:, :O], fx.reference(xref), f"gated input bits {bits} T {T} act {act}")
            assert torch.isnan(y[:, O:]).all()
    with pytest.raises(mlxq.Unsupported):
        layer.linear.encodeGLU(None, gud, stride, 0, y, O + 3, 9)


def test_residual_add_fused_with_the_next_norm(mlxq, oracle):
    # add_rms_norm (Kernels.swift:1141-1175): h += r; y = RMSNorm(h) * w
    g = np.random.default_rng(22)
    for dim, rows, wdt in ((4096, 5, torch.bfloat16), (1000, 1, torch.float32), (64, 3, torch.float16)):
        stride = dim + 4
        h = g.standard_normal((rows, stride)).astype(np.float32)
        r = g.standard_normal((rows, stride)).astype(np.float32)
        w = torch.from_numpy(g.standard_normal(dim).astype(np.float32)).to(wdt)
        hd, rd = torch.from_numpy(h).cuda(), torch.from_numpy(r).cuda()
        yd = torch.zeros((rows, stride), dtype=torch.float32, device="cuda")
        mlxq.addRMSNorm(None, hd, rd, yd, w.cuda(), dim, rows, stride, 1e-6)
        torch.cuda.synchronize()
        href, yref = oracle.add_rms_norm(h[:, :dim], r[:, :dim], w.float().numpy(), 1e-6)
        assert np.array_equal(hd.cpu().numpy()[:, :dim], href)
        assert np.array_equal(hd.cpu().numpy()[:, dim:], h[:, dim:])                    # the padding is not touched
        close(oracle, yd.cpu().numpy()[:, :dim], yref, f"add_rms_norm dim {dim}", 1e-5)


@pytest.mark.parametrize("wdt", [torch.float16, torch.bfloat16, torch.float32])
def test_dense_layers_through_the_same_handle(mlxq, oracle, wdt):
    # dmm (Kernels.swift:938-999): y = x . W^T + bias with W in f32 / f16 / bf16, fp32 accumulation; vector and scalar
    # paths (a K that is not a multiple of 8, strided activations), batches beyond one pass of eight tokens
    g = np.random.default_rng(31)
    for O, K, T, xdt in ((72, 1024, 1, 1), (40, 1000, 5, 0), (33, 36, 20, 2), (16, 4096, 9, 1)):
        w = torch.from_numpy((g.standard_normal((O, K)) * 0.05).astype(np.float32)).to(wdt).cuda()
        bias = torch.from_numpy(g.standard_normal(O).astype(np.float32)).to(wdt).cuda() if O % 2 == 0 else None
        lin = mlxq.Linear(w, None, None, bias, inDim=K, name="dense")
        assert lin.bits == 0
        x = g.standard_normal((T, K)).astype(np.float32)
        xd = as_dtype(x, xdt)
        pad = 8 if K % 8 == 0 else 4                                   # (activation rows stay 16-byte aligned)
        xs = torch.zeros((T, K + pad), dtype=xd.dtype, device="cuda")
        xs[:, :K] = xd
        y = torch.full((T, O + 1), float("nan"), dtype=torch.float32, device="cuda")
        lin.encode(None, xs, K + pad, y, O + 1, T)
        torch.cuda.synchronize()
        ref = oracle.matmul_dense(w.float().cpu().numpy(), xd.float().cpu().numpy(), None if bias is None else bias.float().cpu().numpy())
        close(oracle, y.cpu().numpy()[:, :O], ref, f"dense {wdt} {O}x{K} T {T}", 2e-5)
        assert torch.isnan(y[:, O]).all()
        with pytest.raises(mlxq.Unsupported):
            lin.unpackCodes(None, torch.zeros((O, K), dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("cols,T,pad", [(1, 1, 0), (255, 3, 1), (1021, 700, 0), (1024, 700, 3), (8189, 129, 2)])
def test_activation_product_on_rows_that_are_no_whole_pieces(mlxq, oracle, cols, T, pad):
    # one element per thread where the grid fits on the chip, four where it does not; ragged last blocks
    stride = 2 * cols + pad
    gu = oracle.RNG(cols + T).floats(T * stride).reshape(T, stride)
    out = torch.full((T, cols), float("nan"), device="cuda")
    mlxq.actMul(None, torch.from_numpy(gu).cuda(), stride, cols, T, mlxq.ACT_SILU, out)
    torch.cuda.synchronize()
    g, u = gu[:, :cols].astype(np.float64), gu[:, cols:2 * cols].astype(np.float64)
    ref = g / (1.0 + np.exp(-g)) * u
    assert float(np.max(np.abs(out.cpu().numpy() - ref) / np.maximum(np.abs(ref), 1e-3))) < 2e-6      # expf, a division and two products


@pytest.mark.parametrize("dim", [4, 132, 2048, 4096, 8196, 20480])
def test_add_rms_norm_of_a_row_does_not_depend_on_the_rows_beside_it(mlxq, oracle, dim):
    # many rows take other launch shapes than few: the bits of a row stay the same, and are the oracle's to the rounding of
    # the sum of squares (strands of dim / 1024 terms, then ten pairwise steps: 2^-24 * 20)
    rows = 700
    rng = oracle.RNG(dim)
    h, r, w = (rng.floats(n * dim).reshape(n, dim) for n in (rows, rows, 1))
    stride, outs = dim + 4, []
    for part in (1, 200, rows):
        hd, rd = (torch.full((part, stride), float("nan"), device="cuda") for _ in range(2))
        hd[:, :dim], rd[:, :dim] = torch.from_numpy(h[:part]).cuda(), torch.from_numpy(r[:part]).cuda()
        yd = torch.zeros((part, stride), device="cuda")
        mlxq.addRMSNorm(None, hd, rd, yd, torch.from_numpy(w[0]).cuda(), dim, part, stride, 1e-5)
        torch.cuda.synchronize()
        outs.append((hd[:, :dim].cpu().numpy(), yd[:, :dim].cpu().numpy()))
    for hd, yd in outs[:2]:
        assert np.array_equal(hd, outs[2][0][:len(hd)]) and np.array_equal(yd, outs[2][1][:len(yd)])
    href = h + r
    assert np.array_equal(outs[2][0], href)
    ref = href / np.sqrt((href.astype(np.float64) ** 2).mean(axis=1, keepdims=True) + 1e-5) * w
    assert float(np.max(np.abs(outs[2][1] - ref) / np.maximum(np.abs(ref), 1e-3))) < 20 * 2.0 ** -24


@pytest.mark.parametrize("O,T,x_dtype", [(6143, 3, 0), (6145, 3, 2), (6151, 8, 0), (6145, 11, 1), (4097, 8, 2), (33, 2, 0)])
@pytest.mark.parametrize("w_dtype", [0, 1, 2])
def test_dense_rows_per_warp_at_their_edges(mlxq, oracle, O, T, x_dtype, w_dtype):
    # one and two rows per warp on either side of their bound, odd row counts (the last warp's second row is past the end), a
    # second turn of fewer tokens, a row bias, padded outputs, a ragged last chunk of K
    K, stride = 516 if T == 3 else 520, 536                        # (rows of whole 16-byte pieces and not)
    rng = oracle.RNG(O + T)
    w = as_dtype(rng.floats(O * K).reshape(O, K), w_dtype)
    bias = as_dtype(rng.floats(O), w_dtype)
    x = torch.zeros((T, stride), dtype=TORCH_DT[x_dtype], device="cuda")
    x[:, :K] = as_dtype(rng.floats(T * K).reshape(T, K), x_dtype)
    lin = mlxq.Linear(w, None, None, bias, inDim=K)
    y = torch.full((T, O + 3), float("nan"), device="cuda")
    lin.encode(None, x, stride, y, O + 3, T)
    torch.cuda.synchronize()
    ref = x[:, :K].double() @ w.double().t() + bias.double()
    # fp32 sums of 520 terms in 32 lanes: 17 roundings each and five more, 2^-24 * 22 of the terms' magnitude (below 2 * |y| + 4)
    assert float(((y[:, :O].double() - ref).abs() / (ref.abs() + 4.0)).max()) < 22 * 2.0 ** -23
    assert torch.isnan(y[:, O:]).all()
