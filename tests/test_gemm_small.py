"""The tensor-core kernel for a few dozen tokens (mixfp4_gemm on the stream layout up to 128 rows of x,
mixfp4_gemm_grouped up to 64) against a float64 product with the dequantized weight.

Tolerance: every MMA adds 16 products to an fp32 accumulator with one rounding or truncation, so a chain of K
products is off by at most K / 16 units of 2^-23 of its partial sums, which for these zero-mean inputs are of the
size of the result; a few more for the sums of the chains.  Twice that is allowed."""

import ctypes

import pytest
import torch

import mixfp4_b200 as mx
from mixfp4_b200 import _native as nat
from mixfp4_b200 import linear
from mixfp4_b200 import synth


def tolerance(k: int) -> float:
    return 2 * (k / 16 + 8) * 2.0 ** -23


def weight(n, k, seed):
    w = synth.student_t_weight(n, k, seed).cuda()
    packed = mx.quantize_packed(w)[0].to_stream_layout()
    return packed, packed.dequantize().double()


def check(y, x, wd, k, out):
    ref = x.double() @ wd.T
    rel = ((y.double() - ref).norm() / ref.norm()).item()
    assert rel <= tolerance(k) + (2.0 ** -9 if out == torch.bfloat16 else 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 96, 127, 128])
@pytest.mark.parametrize("n,k", [(16, 16), (17, 128), (130, 96), (128, 256), (1000, 1112), (4240, 640), (2048, 4096), (19000, 384)])
def test_against_float64(m, n, k):
    packed, wd = weight(n, k, n + k)
    x = synth.activations(m, k, m).cuda()
    for out in (torch.float32, torch.bfloat16):
        y = mx.mixfp4_linear(x, packed, out_dtype=out)
        check(y, x, wd, k, out)
    wide = torch.zeros((m, k + 3), dtype=torch.bfloat16, device="cuda")     # rows that a tensor map cannot address
    wide[:, 1:k + 1] = x
    assert torch.equal(mx.mixfp4_linear(wide[:, 1:k + 1], packed), mx.mixfp4_linear(x, packed))
    bare = mx.PackedWeight(packed.codes, packed.scales, None, packed.global_scale, n, k, None, "stream", None)
    assert torch.equal(mx.mixfp4_linear(x, bare), mx.mixfp4_linear(x, packed))       # the kernel builds the decode table
    assert torch.equal(mx.mixfp4_linear(x, packed.to_canonical().to_kernel_layout()), mx.mixfp4_linear(x, packed))
    assert mx.gemm_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m", [17, 48, 64])
@pytest.mark.parametrize("ns,k", [((256, 64, 64), 512), ((4096, 1024, 1000), 4096), ((300, 17), 1112), ((14336, 14336), 640)])
def test_grouped_repeats_and_matches(m, ns, k):
    """One launch for weights that share x, chained to the launch before; thirty launches in a row give the same bits
    (the stages of the weight ring are reused hundreds of times: a release that came too early shows here)."""
    ws = [weight(n, k, i + k) for i, n in enumerate(ns)]
    packs = [p for p, _ in ws]
    x = synth.activations(m, k, m).cuda()
    first = mx.mixfp4_linear_grouped(x, packs, out_dtype=torch.float32)
    for y, (_, wd) in zip(first, ws):
        check(y, x, wd, k, torch.float32)
    runs = [mx.mixfp4_linear_grouped(x, packs, out_dtype=torch.float32, overlap_previous=True) for _ in range(30)]
    assert all(torch.equal(a, b) for run in runs for a, b in zip(run, first))
    assert mx.gemm_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,ns,k", [(8, (200,), 14336), (9, (4096,), 14336), (16, (4096,), 14336), (12, (3000, 3000), 8192),
                                    (16, (128, 100, 16), 9000), (13, (28672,), 8192)])
def test_few_tokens_with_a_large_x(m, ns, k):
    """Up to 16 rows of x that do not fit in the matrix-vector kernel's shared memory: chains of at most 256 products,
    so the error stays at that of the matrix-vector kernels."""
    ws = [weight(n, k, n + k) for n in ns]
    x = synth.activations(m, k, m).cuda()
    ys = mx.mixfp4_linear_grouped(x, [p for p, _ in ws], out_dtype=torch.float32)
    for y, (p, wd) in zip(ys, ws):
        ref = x.double() @ wd.T
        assert ((y.double() - ref).norm() / ref.norm()).item() <= tolerance(256)
        assert torch.equal(mx.mixfp4_linear(x, p).float(), mx.mixfp4_linear(x, p).float())
    runs = [mx.mixfp4_linear_grouped(x, [p for p, _ in ws], out_dtype=torch.float32, overlap_previous=True) for _ in range(10)]
    assert all(torch.equal(a, b) for run in runs for a, b in zip(run, ys))
    assert mx.gemm_status() == 0 and mx.decode_status() == 0


@pytest.mark.gpu
def test_chain_under_dependent_launches_and_graph():
    """Each launch reads the one before it; overlapped launches in a graph give the bits of separate ones."""
    up, _ = weight(2048, 1024, 1)
    down, _ = weight(1024, 2048, 2)
    x = synth.activations(40, 1024, 3).cuda()

    def run(overlap):
        h = x
        for _ in range(4):
            h = mx.mixfp4_linear(mx.mixfp4_linear(h, up, overlap_previous=overlap), down, overlap_previous=overlap)
            h = h / h.float().abs().max().to(h.dtype)
        return h
    want = run(False)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run(True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = run(True)
    torch.cuda.synchronize()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_grouped_entry_checks_its_arguments():
    lib = nat.lib()
    one = ctypes.c_void_p(16)
    seg = (nat.GemvSegment * 1)()
    seg[0].codes, seg[0].global_scale, seg[0].y, seg[0].ldy, seg[0].n = 16, 16, 16, 64, 64
    call = lambda x=one, m=17, ldx=64, k=64, s=seg, count=1, layout=nat.LAYOUT_STREAM, out=nat.F32: lib.mixfp4_gemm_grouped(
        x, m, ldx, k, s, count, layout, out, None, 0, None)
    assert call(layout=nat.LAYOUT_KERNEL) == nat.E_MODE
    assert call(x=None) == nat.E_NULL and call(s=None) == nat.E_NULL
    assert call(m=0) == nat.E_SHAPE and call(m=65) == nat.E_SHAPE and call(count=4) == nat.E_SHAPE and call(ldx=63) == nat.E_SHAPE
    assert call(out=nat.F16) == nat.E_DTYPE
    assert call(x=ctypes.c_void_p(8)) == nat.E_ALIGN and call(ldx=68) == nat.E_ALIGN
    assert call(m=9, x=ctypes.c_void_p(8)) == nat.E_ALIGN and call(m=9, ldx=68) == nat.E_ALIGN
    seg[0].ldy = 63
    assert call() == nat.E_SHAPE
    seg[0].ldy, seg[0].codes = 64, 8
    assert call() == nat.E_ALIGN
    seg[0].codes, seg[0].y = 16, None
    assert call() == nat.E_NULL


def gpu_weight(n, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return mx.quantize_packed((torch.randn((n, k), generator=gen, device="cuda") * 0.02).to(torch.bfloat16))[0]


def errors(y, ref):
    """Error of the whole result and of its worst 128 columns (a tile of the kernel), relative 2-norms."""
    diff = y.double() - ref
    whole = (diff.norm() / ref.norm()).item()
    tiles = [(diff[:, c:c + 128].norm() / ref[:, c:c + 128].norm()).item() for c in range(0, ref.shape[1], 128)]
    return whole, max(tiles)


@pytest.mark.gpu
@pytest.mark.parametrize("m,ns,k", [
    (17, (3000,), 4096), (48, (2048,), 2048), (40, (4096,), 2048), (65, (2048,), 2048), (65, (4096,), 4096), (96, (4096,), 4096), (128, (4096,), 4096), (100, (6144,), 4096),
    (65, (8192,), 8192), (72, (3000,), 8192), (65, (4096,), 14336), (128, (4096,), 14336), (80, (12288,), 14336),
    (128, (12288,), 14336), (65, (8192,), 28672), (96, (8192,), 28672), (128, (8192,), 28672), (48, (12288,), 14336),
    (17, (4096, 1024, 1024), 4096), (48, (4096, 1024, 1024), 4096), (32, (8192, 1024, 1024), 8192),
    (64, (8192, 1024, 1024), 8192), (33, (300, 17), 1112)])
def test_error_is_that_of_the_tiles(m, ns, k):
    """The tensor core's accumulation error grows in proportion to the products summed in one accumulator (after 1024: 7.8e-7
    of the result, after 2048: 1.7e-6), so no accumulator may sum more of them than one of the 128-row tiles that the same
    weight in the canonical layout runs on.  With chains as long the errors agree up to their scatter (2 percent over at least
    17 x 128 outputs; 0.2 of 2^-23 is allowed for the additions of partial sums, whose number differs); a chain twice as
    long doubles the error."""
    packs = [gpu_weight(n, k, n + k + i) for i, n in enumerate(ns)]
    x = synth.activations(m, k, m).cuda()
    ys = mx.mixfp4_linear_grouped(x, [p.to_stream_layout() for p in packs], out_dtype=torch.float32)
    for y, p in zip(ys, packs):
        ref = x.double() @ p.dequantize().double().T
        got, tiles = errors(y, ref), errors(mx.mixfp4_linear(x, p, out_dtype=torch.float32), ref)
        assert all(g <= 1.15 * t + 0.2 * 2.0 ** -23 for g, t in zip(got, tiles))
        assert torch.equal(mx.mixfp4_linear(x, p.to_kernel_layout()), mx.mixfp4_linear(x, p.to_stream_layout()))
    assert mx.gemm_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,own", [(9, True), (16, True), (17, False), (64, False)])
def test_decode_sizes_report_to_the_decode_kernels_word(monkeypatch, m, own):
    """Rows that the decode kernels take (x too large for their shared memory) leave the status word to the library,
    whose own one decode_status() reads; larger batches report to the GEMM's."""
    k = 14336
    packed, wd = weight(300, k, 5)
    x = synth.activations(m, k, m).cuda()
    lib, seen = nat.lib(), []

    class Recorder:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            if name != "mixfp4_gemm_grouped":
                return fn
            return lambda *args: (seen.append(args[8]), fn(*args))[1]
    monkeypatch.setattr(nat, "lib", lambda: Recorder())
    ys = mx.mixfp4_linear_grouped(x, [packed, packed], out_dtype=torch.float32)
    assert len(seen) == 1 and (seen[0] is None) == own
    for y in ys:
        check(y, x, wd, k, torch.float32)
    monkeypatch.undo()
    assert mx.decode_status() == 0 and mx.gemm_status() == 0


@pytest.mark.gpu
def test_no_workspace_is_kept_for_partial_sums_that_nothing_writes():
    m, n, k = 128, 4096, 14336
    packed = gpu_weight(n, k, 1).to_stream_layout()
    x = synth.activations(m, k, m).cuda()
    linear._workspaces.clear()
    y = mx.mixfp4_linear(x, packed)
    assert sum(w.numel() for w in linear._workspaces.values()) <= m * k * 2 + 4096
    mx.mixfp4_linear(x, packed.to_canonical())                       # the tiles: room for their partial sums
    assert torch.equal(mx.mixfp4_linear(x, packed), y)
