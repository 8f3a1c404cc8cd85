"""Branches of the format kernels that small tests do not reach: bf16 tiles that arrive by TMA (several per CTA, ragged row
counts), and the re-encoding that brings its count to the host by itself (slots used again and by several threads)."""
import threading

import numpy as np
import pytest

import fp8_quant_matmul_b200 as f

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", ["rowwise", "block"])
@pytest.mark.parametrize("shape", [(16, 128), (144, 384), (128, 8192), (2064, 4096), (7184, 1152)],      # up to 544 tiles on 444 CTAs
                         ids=lambda s: "x".join(map(str, s)))
def test_bf16_quantiser_equals_the_fp32_one_on_the_same_values(kind, shape):
    g = torch.Generator(device="cuda").manual_seed(shape[0] + shape[1])
    X = (torch.randn(shape, generator=g, device="cuda") * torch.exp(torch.randn(shape[1], generator=g, device="cuda"))).bfloat16()
    X[3].zero_()
    quantize = f.quantize_rowwise if kind == "rowwise" else f.quantize_block
    q, s = quantize(X)
    q32, s32 = quantize(X.float())
    f.last_device_status()
    assert torch.equal(q, q32) and torch.equal(s, s32)


@pytest.mark.parametrize("n", [16, 4096 + 5, 148 * 8 * 256 * 16 * 2 + 48])
def test_reencode_counts_every_inexact_byte_in_every_call(n):
    rng = np.random.default_rng(n)
    b = rng.integers(0, 256, n, dtype=np.uint8)
    want = int(((b & 0x7F) < 16).astype(np.int64) @ (b & 1))           # odd multiples of 2^-10 below 2^-6, either sign
    src = torch.from_numpy(b).cuda()
    first, got = f.fnuz_to_fn_device(src)
    assert got == want
    for _ in range(3):                                                  # the slot is clean again
        again, got = f.fnuz_to_fn_device(src)
        assert got == want and torch.equal(first, again)


def test_reencode_from_several_threads_and_streams():
    srcs = [torch.randint(0, 256, (100000 + 16 * i,), dtype=torch.uint8, device="cuda") for i in range(8)]
    want = [f.fnuz_to_fn_device(s)[1] for s in srcs]
    torch.cuda.synchronize()
    got = [[] for _ in srcs]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got[i].append(f.fnuz_to_fn_device(srcs[i])[1])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(srcs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[w] * 20 for w in want]


def test_reencode_is_refused_under_capture_and_works_afterwards():
    src = torch.randint(0, 256, (100000,), dtype=torch.uint8, device="cuda")
    dst, want = f.fnuz_to_fn_device(src)
    copy = torch.zeros_like(src)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        copy.copy_(src)
        for _ in range(80):                                             # more often than there are slots
            with pytest.raises(f.Fp8bsError) as error:
                f.fnuz_to_fn_device(src, copy)
            assert error.value.code == -7
    graph.replay()
    again, got = f.fnuz_to_fn_device(src)
    assert got == want and torch.equal(again, dst) and torch.equal(copy, src)


def test_reencode_by_more_callers_than_there_are_slots():
    callers = 96
    srcs = [torch.randint(0, 256, (50000 + 16 * i,), dtype=torch.uint8, device="cuda") for i in range(callers)]
    want = [f.fnuz_to_fn_device(s) for s in srcs]
    streams = [torch.cuda.Stream() for _ in range(24)]
    torch.cuda.synchronize()
    got = [None] * callers
    together = threading.Barrier(callers)

    def work(i):
        with torch.cuda.stream(streams[i % len(streams)]):
            together.wait(60)
            for _ in range(5):
                got[i] = f.fnuz_to_fn_device(srcs[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(callers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(g is not None and g[1] == w[1] and torch.equal(g[0], w[0]) for g, w in zip(got, want))
