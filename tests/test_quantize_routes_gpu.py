"""The quantizer's one-pass routes against the separate passes they stand for, bit for bit: the stream-layout
quantizer, the fused region selection and the packed fp32 path, over odd sizes, strides, types and special values."""

import numpy as np
import pytest
import torch

import oracle
import mixfp4_b200 as mx
from mixfp4_b200 import _native as nat
from mixfp4_b200 import quant as Q
from mixfp4_b200 import synth

pytestmark = pytest.mark.gpu
DTYPES = [torch.bfloat16, torch.float16, torch.float32]


def bits(t: torch.Tensor) -> torch.Tensor:
    return t.contiguous().view(torch.int16 if t.element_size() == 2 else torch.int32)


def tensor(rows, k, dtype, seed, scale=1.0):
    x = synth.activations(rows, k, seed, outlier_fraction=0.02).float() * scale
    x[0, : min(k, 16)] = 0.0                     # an all-zero block
    x[-1, -1] = -0.0
    if rows > 2:
        x[1, :] *= 2e-5                          # blocks whose scales are subnormal E4M3 numbers
    return x.to(dtype).cuda()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,k", [(1, 16), (16, 128), (17, 130), (33, 1000), (5, 4100), (300, 257)])
@pytest.mark.parametrize("mode", ["oracle16", "all_e2m1", "all_e0m3"])
def test_stream_quantizer_equals_quantize_then_repack(dtype, rows, k, mode):
    x = tensor(rows, k, dtype, 3 * rows + k, 0.01)
    want = mx.quantize_packed(x, mode=mode)[0].to_stream_layout()
    got = Q.quantize_stream(x, mode=mode)
    assert torch.equal(got.codes, want.codes) and torch.equal(got.lut, want.lut)
    assert torch.equal(bits(got.global_scale), bits(want.global_scale))
    view = torch.empty((rows, k + 3), dtype=dtype, device="cuda")[:, 1:k + 1]      # unaligned rows
    view.copy_(x)
    assert torch.equal(Q.quantize_stream(view, mode=mode).codes, want.codes)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("role,mode", [("weight_b", m) for m in ("k32_row", "k64_row", "n2k64", "n4k64", "n8k64", "n16k64", "n32k64", "n64k64", "n8k16")]
                         + [("activation_a", "m16k16"), ("activation_a", "m32k64")])
@pytest.mark.parametrize("rows,k", [(1, 160), (64, 512), (70, 1111), (129, 4100)])
def test_fused_regions_equal_the_three_passes(dtype, role, mode, rows, k):
    x = tensor(rows, k, dtype, rows + k)
    region = Q.region_shape(mode, role)
    want = mx.quantize_packed(x, mode=mode, want_dequant=True, region=region)[1]
    got = mx.quant_mixfp4_granularity(x, format_region=mode, operand_role=role)
    assert torch.equal(bits(got), bits(want))
    view = torch.empty((rows, k + 5), dtype=dtype, device="cuda")[:, 1:k + 1]
    view.copy_(x)
    assert torch.equal(bits(mx.quant_mixfp4_granularity(view, format_region=mode, operand_role=role)), bits(want))


@pytest.mark.parametrize("scale", [1e-6, 0.02, 37.0, 5e4])
def test_fp32_path_against_oracle(scale):
    """The packed path takes tensor scales up to 1 (a maximum of 2688), the IEEE path the rest."""
    w = (synth.student_t_weight(257, 1040, 11).float() * 1.2345 * scale)
    ref = oracle.quantize(w.numpy())
    packed, dq, _ = mx.quantize_packed(w.cuda(), want_dequant=True)
    assert np.array_equal(packed.codes.cpu().numpy(), ref.codes)
    assert np.array_equal(packed.scales.cpu().numpy(), ref.scales)
    assert np.array_equal(packed.fmt.cpu().numpy(), ref.fmt)
    assert np.array_equal(dq.cpu().numpy().view(np.uint32), np.ascontiguousarray(oracle.dequant(ref, "f32")).view(np.uint32))


@pytest.mark.parametrize("dtype", DTYPES)
def test_nan_elements_leave_other_blocks_alone(dtype):
    """A NaN takes the largest level of its block (as it did before the packed fp32 path); the other
    blocks are those of the tensor without it."""
    x = tensor(8, 256, dtype, 5)
    y = x.clone()
    y[3, 40] = float("nan")
    a, b = mx.quant_mixfp4_granularity(x), mx.quant_mixfp4_granularity(y)
    mask = torch.ones_like(x, dtype=torch.bool)
    mask[3, 32:48] = False
    assert torch.equal(bits(a)[mask], bits(b)[mask]) and torch.isfinite(b).all()


def test_rotation_with_maximum():
    for dtype, k in ((torch.bfloat16, 512), (torch.float16, 300), (torch.float32, 256)):
        x = tensor(37, k, dtype, k)
        amax = torch.empty(1, device="cuda")
        y = mx.apply_transform(x, "H128")
        from mixfp4_b200 import rotation
        z = rotation.apply_transform(x, "H128", amax=amax)
        assert torch.equal(bits(y), bits(z)) and amax.item() == y.float().abs().max().item()


def test_routes_refuse_bad_arguments():
    lib, p = nat.lib(), torch.empty(4096, dtype=torch.uint8, device="cuda").data_ptr()
    assert lib.mixfp4_quantize_stream(None, 0, 16, 128, 128, 0, p, p, p, None, None) == -1
    assert lib.mixfp4_quantize_stream(p, 0, 16, 128, 64, 0, p, p, p, None, None) == -2
    assert lib.mixfp4_quantize_stream(p, 7, 16, 128, 128, 0, p, p, p, None, None) == -4
    assert lib.mixfp4_quantize_stream(p, 0, 16, 128, 128, 3, p, p, p, None, None) == -5
    assert lib.mixfp4_quantize_stream(p, 0, 16, 128, 128, 0, p, p + 8, p, None, None) == -3
    assert lib.mixfp4_fake_quantize_regions(p, 0, 16, 128, 128, 3, 4, p, p + 1, 128, None) == -5
    assert lib.mixfp4_fake_quantize_regions(p, 0, 16, 128, 128, 8, 4, p, p, 128, None) == -2
    assert lib.mixfp4_fake_quantize_regions(p, 0, 16, 64, 64, 8, 4, p, p + 2048, 64, None) == -5
