"""Calls of two to sixteen tokens have two kernels, the token-major one (qmv_tok.cuh) and the tensor-memory one (qmv_tc.cuh):
which of them takes a call, and the tensor-memory kernel at its edges, against the oracle.  MLXQ_DECODE is read at every call."""
import pytest
import torch

from helpers import TENSOR_MEMORY_CALLS, TORCH_DT, DevLayer, as_dtype

pytestmark = pytest.mark.gpu


def forward(layer, x, T):
    O = layer.linear.outDim
    y = torch.full((T, O), float("nan"), device="cuda")
    layer.linear.encode(None, x, layer.linear.inDim, y, O, T)
    torch.cuda.synchronize()
    return y


def test_a_kernel_is_chosen_by_its_name_only(mlxq, oracle, monkeypatch):
    # 12 fp32 tokens: the tensor-memory kernel's; a value that names no kernel changes nothing
    K, O, T = 2048, 264, 12
    fx = oracle.QuantFixture(O=O, K=K, bits=4, gs=64, scale_type=oracle.BF16, seed=3)
    layer = DevLayer.from_fixture(mlxq, fx)
    x = as_dtype(oracle.RNG(5).floats(T * K).reshape(T, K), 0)
    got = {}
    for mode in (None, "", "another", "tc", "tok", "cuda"):
        if mode is None:
            monkeypatch.delenv("MLXQ_DECODE", raising=False)
        else:
            monkeypatch.setenv("MLXQ_DECODE", mode)
        got[mode] = forward(layer, x, T)
    for mode in ("", "another", "tc"):
        assert torch.equal(got[mode], got[None]), f"MLXQ_DECODE={mode!r} changed the kernel"
    for mode in ("tok", "cuda"):
        assert not torch.equal(got[mode], got[None]), f"MLXQ_DECODE={mode!r} was not obeyed"
        assert oracle.max_rel_err(got[mode].cpu().numpy(), fx.reference(x.cpu().numpy())) < 1e-4


@pytest.mark.parametrize("x_dtype,T", [(0, 4), (0, 8), (0, 12), (2, 13)])
def test_shards_keep_to_the_kernels_of_the_fused_gather(mlxq, oracle, monkeypatch, x_dtype, T):
    # the fused gather runs on the token-major kernel (or what stands in for it), the gathers after the call must give the
    # same bits: rows of 4096 codes, where a whole layer's batches take the tensor-memory kernel
    K, O, bits, gs = 4096, 1024, 4, 64
    fx = oracle.QuantFixture(O=O, K=K, bits=bits, gs=gs, scale_type=oracle.BF16, seed=T)
    full = DevLayer.from_fixture(mlxq, fx)
    shard = mlxq.Linear.shard(full.w, full.s, full.b, None, inDim=K, rank=1, nranks=2, full=True, name="shard", device=0)
    x = as_dtype(oracle.RNG(T).floats(T * K).reshape(T, K), x_dtype)
    got = {}
    for mode in (None, "tok"):
        if mode is None:
            monkeypatch.delenv("MLXQ_DECODE", raising=False)
        else:
            monkeypatch.setenv("MLXQ_DECODE", mode)
        y = torch.full((T, O // 2), float("nan"), device="cuda")
        shard.encode(None, x, K, y, O // 2, T)
        torch.cuda.synchronize()
        got[mode] = y
    assert torch.equal(got[None], got["tok"])
    assert oracle.max_rel_err(got[None].cpu().numpy(), fx.reference(x.float().cpu().numpy())[:, O // 2:]) < 1e-3


def codes_of(w, bits, K):
    """Packed words -> codes [rows, K]"""
    b = w.view(torch.uint8).view(w.shape[0], -1)
    if bits in (2, 4, 8):
        return torch.stack([(b >> at) & ((1 << bits) - 1) for at in range(0, 8, bits)], -1).reshape(-1, K)
    one = torch.stack([(b >> i) & 1 for i in range(8)], -1).reshape(-1, K, bits)
    return (one << torch.arange(bits, dtype=torch.uint8, device=w.device)).sum(-1, dtype=torch.uint8)


@pytest.mark.parametrize("bits,gs,K,O,T,x_dtype", [(8, 32, 12288, 512, 16, 2), (8, 32, 14336, 512, 11, 1), (8, 64, 12288, 8192, 13, 2),
                                                   (6, 32, 12288, 512, 13, 2), (5, 32, 14336, 512, 5, 2), (4, 64, 4096, 512, 6, 0), (8, 128, 12288, 512, 16, 1)])
def test_no_less_exact_than_the_kernels_before(mlxq, monkeypatch, bits, gs, K, O, T, x_dtype):
    # the error against 64 bits, with the kernel that the dispatch takes and without the tensor-memory kernel.  A norm over
    # O * T >= 2560 outputs with independent roundings is known to 1 / sqrt(2 * 2560) = 1.4 %: three times that.
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + T)
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (O, K * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = (torch.randn((O, K // gs), device="cuda", generator=gen).abs() * 0.002 + 1e-4).to(torch.bfloat16)
    b = (-float(1 << (bits - 1)) * s.float()).to(torch.bfloat16)
    lin = mlxq.Linear(w, s, b, None, inDim=K)
    x = torch.randn((T, K), device="cuda", generator=gen).to(TORCH_DT[x_dtype])
    ref = x.double() @ (codes_of(w, bits, K).double() * s.double().repeat_interleave(gs, 1) + b.double().repeat_interleave(gs, 1)).T
    err = {}
    for mode in (None, "tok"):
        if mode is None:
            monkeypatch.delenv("MLXQ_DECODE", raising=False)
        else:
            monkeypatch.setenv("MLXQ_DECODE", mode)
        y = torch.full((T, O), float("nan"), device="cuda")
        lin.encode(None, x, K, y, O, T)
        torch.cuda.synchronize()
        err[mode] = ((y.double() - ref).norm() / ref.norm()).item()
    assert err[None] <= 1.05 * err["tok"], err


@pytest.mark.parametrize("call", TENSOR_MEMORY_CALLS, ids=str)
def test_tensor_memory_kernel_at_its_edges(mlxq, monkeypatch, call):
    # against the same sums in 64 bits; x and y with padding, which must be neither read nor written
    bits, gs, K, rows, T, x_dtype, offset, with_bias = call
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + T + bits)

    def behind(t):
        flat = torch.zeros(t.numel() + offset, dtype=t.dtype, device="cuda")
        flat[offset:] = t.reshape(-1)
        return flat[offset:].view(t.shape)

    lins, refs, keep = [], [], []
    x = torch.full((T, K + 8), float("nan"), device="cuda", dtype=TORCH_DT[x_dtype])
    x[:, :K] = torch.randn((T, K), device="cuda", generator=gen).to(TORCH_DT[x_dtype])
    for o in rows:
        w = torch.randint(-(1 << 31), (1 << 31) - 1, (o, K * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
        s = (torch.randn((o, K // gs), device="cuda", generator=gen).abs() * 0.002 + 1e-4).to(torch.float16 if bits % 2 else torch.bfloat16)
        b = (-float(1 << (bits - 1)) * s.float()).to(s.dtype)
        bias = torch.randn(o, device="cuda", generator=gen).to(s.dtype) if with_bias else None
        keep.append((w, behind(s), behind(b), bias))
        lins.append(mlxq.Linear(*keep[-1], inDim=K))
        wd = codes_of(w, bits, K).double() * s.double().repeat_interleave(gs, 1) + b.double().repeat_interleave(gs, 1)
        refs.append(x[:, :K].double() @ wd.T + (bias.double() if with_bias else 0.0))
    O = sum(rows)
    ref = torch.cat(refs, 1)
    y = torch.full((T, O + 3), float("nan"), device="cuda")
    monkeypatch.setenv("MLXQ_DECODE", "tc")
    for _ in range(2):
        if len(lins) == 1:
            lins[0].encode(None, x, K + 8, y, O + 3, T)
        else:
            mlxq.Linear.encodeFusedDecode(None, lins, x, y, K + 8, O + 3, T)
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    assert torch.isnan(y[:, O:]).all()
    # a rounding of 2^-24 for each of the K / gs groups added up, of a running sum that holds up to the result's magnitude and, per
    # group, of products some times larger; an fp32 activation's two parts leave 2^-22 of a product
    bar = 2.0 ** -24 * (2.0 * (K / gs) ** 0.5 + 2.0)
    err = ((y[:, :O].double() - ref).norm() / ref.norm()).item()
    assert err < bar, f"{err} of the result, bar {bar}"
    # no single output further off than such a sum can be: six deviations
    worst = ((y[:, :O].double() - ref).abs().max() / ref.pow(2).mean().sqrt()).item()
    assert worst < 6 * bar, f"{worst} of the root mean square"
    for dtype in (torch.float16, torch.bfloat16):                  # 16-bit outputs: the same sums, rounded once
        y16 = torch.full((T, O + 3), float("nan"), device="cuda", dtype=dtype)
        if len(lins) == 1:
            lins[0].encode(None, x, K + 8, y16, O + 3, T)
        else:
            mlxq.Linear.encodeFusedDecode(None, lins, x, y16, K + 8, O + 3, T)
        torch.cuda.synchronize()
        assert torch.equal(y16[:, :O], y[:, :O].to(dtype)) and torch.isnan(y16[:, O:]).all()


@pytest.mark.parametrize("bits,K,O,T,x_dtype", [(4, 4096, 24576, 6, 0), (4, 4096, 24576, 16, 1), (3, 4096, 11008, 16, 0), (8, 12288, 4096, 8, 0)])
def test_tensor_memory_kernel_repeats_bit_for_bit_at_full_size(mlxq, monkeypatch, bits, K, O, T, x_dtype):
    # sums are formed in a fixed order, and every wait before a tensor-memory store is by one polling lane: twelve calls of full
    # size, one right after the other and with dependent launches in flight, give the same bits
    gen = torch.Generator(device="cuda")
    gen.manual_seed(O + T)
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (O, K * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    s = (torch.rand((O, K // 64), device="cuda", generator=gen) * 0.004).to(torch.bfloat16)
    lin = mlxq.Linear(w, s, (-float(1 << (bits - 1)) * s.float()).to(torch.bfloat16), None, inDim=K)
    x = torch.randn((T, K), device="cuda", generator=gen).to(TORCH_DT[x_dtype])
    monkeypatch.setenv("MLXQ_DECODE", "tc")
    ys = [torch.full((T, O), float("nan"), device="cuda") for _ in range(12)]
    for y in ys:
        lin.encode(None, x, K, y, O, T)
    torch.cuda.synchronize()
    mlxq.streamStatus(None, 0)
    assert torch.isfinite(ys[0]).all()
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
