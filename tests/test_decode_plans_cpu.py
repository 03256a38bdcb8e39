"""The decode kernels' planners, run on the host: what they place lies inside the shared memory they ask for."""
import importlib.util
import os
import subprocess

import pytest

from helpers import TENSOR_MEMORY_CALLS

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PKG = os.path.join(ROOT, "mlx-runner_b200")

SMEM_OPT_IN = 227 * 1024
NAMED, TOKEN_MAJOR, CLUSTER, SCALED_CLUSTER, HALVES, GENERAL, OTHER = range(7)       # enum TcInstead


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    """calls -> planned layouts: lists of integers, one per planner (see decode_plans.cu)."""
    spec = importlib.util.spec_from_file_location("mlxq_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build()
    exe = str(tmp_path_factory.mktemp("plans") / "decode_plans")
    objs = [os.path.join(build.OBJ, o) for (_, o, _) in build.UNITS]
    subprocess.run([build._nvcc()] + build.COMMON + ["-I", build.CSRC, os.path.join(HERE, "decode_plans.cu"), "-o", exe] + objs + ["-ldl"], check=True)

    def run(calls, *args):
        text = "\n".join(" ".join(str(v) for v in c) for c in calls)
        out = subprocess.run([exe, *args], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
        assert len(out) == len(calls)
        return [[[int(v) for v in part.split()] for part in line.split("|")] for line in out]

    return run


def test_no_row_length_leaves_the_shared_memory_asked_for(plans):
    # a layer may have rows of up to 2^30 codes: lengths at which a 32-bit size of 2, 4, 8 ... 64 bytes a code wraps around,
    # lengths around them, and a walk over the rest
    lengths = {65075328, 33554432, 1 << 30}
    for shift in range(20, 31):
        for num in range(1, 16):
            at = (num << shift) // 4
            lengths.update(at + d * 128 for d in (-80, -3, -1, 0, 1, 2, 40) if 1024 <= at + d * 128 <= 1 << 30)
    lengths.update(range(1024, 1 << 18, 640))
    lengths.update(range(1 << 18, 1 << 30, 1021 * 1024))
    calls = [(bits, gs, k // 128 * 128, rows, tokens, split, NAMED) for k in sorted(lengths)
             for bits, gs, rows, tokens, split in ((4, 64, 128, 16, 2), (8, 32, 40, 8, 2), (4, 128, 4096, 16, 1), (2, 64, 24, 3, 2), (6, 32, 64, 6, 2))]
    served = 0
    for call, (tc, *others) in zip(calls, plans(calls)):
        smem, kz, stages, depth, off_x, off_xsum, off_red, off_bars, *_ = tc
        if smem:
            served += 1
            bits, gs, k, rows, tokens, split, _ = call
            slice_ = -(-stages // kz)
            x_bytes = slice_ * 2 * split * (1024 if tokens <= 8 else 2048)
            assert stages == k // 128 and depth >= 3 and smem <= SMEM_OPT_IN, call
            assert 0 < off_x and off_x + x_bytes <= off_xsum < off_red < off_bars < smem, f"{call}: {tc}"
        for plan in others:
            if plan[0]:
                served += 1
                assert plan[0] <= SMEM_OPT_IN and all(a <= b for a, b in zip([1] + plan[1:], plan[1:] + [plan[0]])), f"{call}: {plan}"
    assert served > 300


def test_clusters_are_the_ones_that_the_device_holds(plans):
    calls = [(4, 64, k, rows, tokens, 2, NAMED) for k in (1024, 4096, 12288) for rows in (128, 4096, 40960) for tokens in (2, 6, 16)]
    for args, room in (((), {1: 296, 2: 148, 4: 71, 8: 33}), (("part",), {1: 40, 2: 20, 4: 10})):
        cuts = set()
        for call, (tc, *_) in zip(calls, plans(calls, *args)):
            if tc[0]:
                kz, clusters, n_blocks = tc[1], tc[-2], tc[-1]
                assert kz in room and 1 <= clusters <= min(room[kz], n_blocks), f"{call}: {tc}"
                cuts.add(kz)
        assert cuts >= set(room) - {1, 2}, cuts


# (bits, group, K, rows, tokens, fp16 parts per activation), what the call runs on otherwise, and whether the tensor-memory kernel takes it
@pytest.mark.parametrize("call,instead,taken", [
    # 3 bits, 8 fp16 tokens of 4096 codes (64 KB staged by a CTA of the token-major kernel): the tallest layers stay there
    ((3, 64, 4096, 11008, 8, 1), TOKEN_MAJOR, True), ((3, 64, 4096, 15368, 8, 1), TOKEN_MAJOR, False), ((2, 128, 4096, 16384, 8, 1), TOKEN_MAJOR, False),
    # the batch of six of a 4-bit decode step, its 6-bit vocabulary head, and its neighbours in tokens
    ((4, 64, 4096, 24576, 6, 2), TOKEN_MAJOR, True), ((4, 64, 4096, 4096, 6, 2), TOKEN_MAJOR, True), ((4, 64, 12288, 4096, 6, 2), CLUSTER, True),
    ((6, 64, 4096, 151936, 6, 2), TOKEN_MAJOR, False), ((4, 64, 4096, 24576, 4, 2), TOKEN_MAJOR, False), ((4, 64, 2048, 24576, 6, 2), TOKEN_MAJOR, False),
    # on either side of the rows that a limit stands at
    ((5, 64, 4096, 3072, 5, 1), TOKEN_MAJOR, True), ((5, 64, 4096, 3080, 5, 1), TOKEN_MAJOR, False),
    ((8, 64, 4096, 3072, 6, 2), TOKEN_MAJOR, True), ((8, 64, 4096, 3080, 6, 2), TOKEN_MAJOR, False),
    # two launches of half the tokens; not vocabulary-sized layers at 8 bits on rows that cut badly
    ((8, 64, 2560, 32768, 16, 2), HALVES, True), ((8, 64, 2560, 32776, 16, 2), HALVES, False), ((4, 64, 2560, 151936, 16, 2), HALVES, True),
    # in the place of kernels without tensor cores, from two fp32 (three, of the general plan) or five 16-bit tokens on
    ((2, 32, 512, 4096, 2, 2), OTHER, True), ((2, 32, 512, 4096, 3, 2), GENERAL, True), ((2, 32, 512, 4096, 2, 2), GENERAL, False), ((2, 32, 512, 4096, 5, 1), OTHER, True), ((2, 32, 512, 4096, 4, 1), OTHER, False),
    # 8 bits with 16-bit activations: while the sums are short enough
    ((8, 32, 8192, 4096, 16, 1), OTHER, True), ((8, 32, 12288, 4096, 16, 1), OTHER, False), ((8, 64, 14336, 4096, 16, 1), OTHER, True),
    # what the kernel cannot serve
    ((4, 64, 4096 + 64, 4096, 6, 2), NAMED, False), ((4, 64, 4096, 4096, 17, 2), NAMED, False), ((4, 64, 4096, 4096, 1, 2), NAMED, False),
])
def test_which_small_batches_the_tensor_memory_kernel_takes(plans, call, instead, taken):
    assert (plans([call + (instead,)])[0][0][0] > 0) == taken


def test_every_compiled_kernel_is_one_that_the_dispatch_takes(plans):
    # (width, tokens compiled for, parts): two fp32 tokens at 6 and 8 bits and four 16-bit ones and fewer are not compiled, not even
    # where the kernel is named; every other instance is reached by some call
    calls = [(bits, gs, k, rows, tokens, split, instead) for bits in (2, 3, 4, 5, 6, 8) for gs in (32, 64) for k in (2048, 4096, 8192, 11008, 12288)
             for rows in (1024, 4096) for tokens in (2, 3, 4, 5, 8, 9, 16) for split in (1, 2) for instead in (NAMED, TOKEN_MAJOR, OTHER)]
    named, chosen = set(), set()
    for (bits, _, _, _, tokens, split, instead), (tc, *_) in zip(calls, plans(calls)):
        if tc[0]:
            (named if instead == NAMED else chosen).add((bits, 2 if tokens <= 2 else 4 if tokens <= 4 else 8 if tokens <= 8 else 16, split))
    assert named == chosen
    assert len(named) == 34 and not any(split == 1 and ntk <= 4 for _, ntk, split in named)


def test_the_edges_that_the_gpu_tests_reach(plans):
    # every cut with six rounds of blocks and more in at least one CTA (the sums' buffers are used again from the third on), every
    # depth of the ring, an odd number of groups in a slice, fewer stages than turns that only fetch, all compiled batches
    reached = [plans([(bits, gs, k, sum(rows), tokens, 2 if x_dtype == 0 else 1, NAMED)])[0][0]
               for bits, gs, k, rows, tokens, x_dtype, _, _ in TENSOR_MEMORY_CALLS]
    assert all(tc[0] for tc in reached)
    assert {tc[1] for tc in reached if tc[-1] > 5 * tc[-2]} == {1, 2, 4, 8}
    assert {tc[3] for tc in reached} == {3, 4, 6, 8}
    assert any(tc[0] > 113 * 1024 for tc in reached)
    assert any(k // gs % 2 for _, gs, k, *_ in TENSOR_MEMORY_CALLS) and min(tc[2] // tc[1] for tc in reached) == 1
    assert {(2 if t <= 2 else 4 if t <= 4 else 8 if t <= 8 else 16, 2 if x == 0 else 1) for *_, t, x, _, _ in TENSOR_MEMORY_CALLS} == \
        {(2, 2), (4, 2), (8, 2), (16, 2), (8, 1), (16, 1)}
