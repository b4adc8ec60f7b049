"""Edges of the tensor-core SC conv: tiles of 320 candidates, units of 160, channel words per pipeline step, rows of the
patch, and the choice between the standard and the compact activation grid.  Integer work: bit-exact against the
direct kernel, which the oracle tests cover."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(ops, n, c, h, w, co, k, stride, pad, own_pad, L, or_n, nhwc, dtype, border=0.0):
    g = torch.Generator(device="cuda").manual_seed(n * 1000003 + c * 1009 + h * 31 + co)
    x = (torch.randn(n, c, h, w, device="cuda", generator=g) * 0.45).clamp(0, 1).to(dtype)
    wt = (torch.randn(co, c, k, k, device="cuda", generator=g) * 0.2).clamp(-1, 1)
    wt[0] = float("nan")  # quantises like the two clamps of the reference leave it
    if not own_pad and pad:
        x = torch.nn.functional.pad(x, (pad,) * 4, value=border)
    fmt = torch.channels_last if nhwc else torch.contiguous_format
    x, wt = x.contiguous(memory_format=fmt), wt.contiguous(memory_format=fmt)
    out = []
    for kernel in ("tensor", "direct"):
        ops.set_conv_kernel(kernel)
        try:
            p = pad if own_pad else 0
            out.append(ops.conv2d_generic_general_split_acc(x, wt, L, -1, 16, (p, p), (stride, stride), (7, 8, 1),
                                                            or_n - 1, 1, True, False))
            assert ops.workspace_status() == 0
        finally:
            ops.set_conv_kernel("auto")
    for a, b in zip(*out):
        assert torch.equal(a, b), f"{(a != b).sum().item()} counts differ"


@pytest.mark.parametrize("pixels", [1, 159, 160, 161, 319, 320, 321, 640, 961])
@pytest.mark.parametrize("nhwc", [True, False])
def test_tile_and_unit_edges(ops, pixels, nhwc):
    _both(ops, 1, 32, 1, pixels, 64, 1, 1, 0, True, 32, 2, nhwc, torch.float32)


@pytest.mark.parametrize("c", [1, 32, 33, 64, 65, 96, 128, 160, 256, 288, 512])
@pytest.mark.parametrize("k", [1, 3])
def test_channel_words_per_step(ops, c, k):
    _both(ops, 2, c, 9, 11, 40, k, 1, k // 2, True, 64, 3, True, torch.float16)


@pytest.mark.parametrize("co", [1, 2, 10, 63, 64, 65, 72, 128, 130])
@pytest.mark.parametrize("nhwc", [True, False])
def test_output_channels_and_layouts(ops, co, nhwc):
    _both(ops, 3, 40, 13, 17, co, 3, 1, 1, True, 32, 1, nhwc, torch.bfloat16)


@pytest.mark.parametrize("or_n,L", [(1, 128), (4, 256 // 2), (60, 128), (500, 128), (3000, 16)])
def test_limits_and_long_streams(ops, or_n, L):
    _both(ops, 2, 64, 10, 10, 64, 3, 1, 1, True, L, or_n, True, torch.float32)


@pytest.mark.parametrize("k,stride,h,w", [(3, 2, 112, 120), (3, 2, 200, 9), (2, 2, 30, 31), (2, 1, 30, 31),
                                           (1, 2, 57, 58), (3, 1, 5, 400)])
def test_strides_and_patch_rows(ops, k, stride, h, w):
    _both(ops, 1, 48, h, w, 64, k, stride, k // 2, True, 32, 2, True, torch.float16)


@pytest.mark.parametrize("border", [0.0, 0.5])
@pytest.mark.parametrize("n,c,co", [(64, 128, 512), (1, 64, 64)])
def test_caller_padded_layers(ops, n, c, co, border):
    """A zero border (compact grid) and one that is not (found out by the expand launch)."""
    _both(ops, n, c, 7, 7, co, 3, 1, 1, False, 32, 2, True, torch.float16, border)
    _both(ops, n, c, 7, 7, co, 3, 1, 1, False, 32, 2, False, torch.float32, border)


@pytest.mark.parametrize("on", ["input", "weight"])
def test_output_on_an_operands_storage(ops, on):
    """``out`` tensors that share the activation's or the weight's memory: both are read before an output is written,
    although the outputs of so small a layer are cleared by the launch that reads the operands."""
    g = torch.Generator(device="cuda").manual_seed(5)
    h = 56 if on == "input" else 3
    fmt = torch.channels_last
    x = (torch.randn(1, 64, h, h, device="cuda", generator=g) * 0.45).clamp(0, 1).half().contiguous(memory_format=fmt)
    wt = (torch.randn(64, 64, 3, 3, device="cuda", generator=g) * 0.2).clamp(-1, 1).half().contiguous(memory_format=fmt)
    args = (32, -1, 16, (1, 1), (1, 1), (7, 8, 1), 1, 1, True, False)
    want = ops.conv2d_generic_general_split_acc(x, wt, *args)
    if on == "input":
        shared = x.view(torch.int16)
    else:
        shared = wt.permute(0, 2, 3, 1).reshape(-1)[:64 * h * h].view(torch.int16).view(1, h, h, 64).permute(0, 3, 1, 2)
        assert shared.data_ptr() == wt.data_ptr()
    got = ops.conv2d_generic_general_split_acc(x, wt, *args, out=(shared, torch.empty_like(shared)))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
