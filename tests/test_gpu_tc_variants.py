"""Edges of the tensor-core SC conv: tiles of 320 candidates, units of 160, channel words per pipeline step, rows of the
patch, and the choice between the standard and the compact activation grid.  Integer work: bit-exact against the
direct kernel, which the oracle tests cover."""
import pytest
import torch

from test_gpu_sc_conv import _torch_loop_linear_counts

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


@pytest.mark.parametrize("lfsr", [1, 2])
@pytest.mark.parametrize("xnor", [True, False])
@pytest.mark.parametrize("nhwc", [True, False])
def test_shortest_registers(ops, oracle, lfsr, xnor, nhwc):
    """Explicit 1- and 2-bit registers, whose cycle is one state longer than the 2^l - 1 of the others, on the merged
    expand launch (32 and 64 slots) and the separate ones (128)."""
    g = torch.Generator().manual_seed(lfsr)
    x = torch.rand(2, 40, 7, 9, generator=g)
    wt = (torch.randn(70, 40, 3, 3, generator=g) * 0.5).clamp(-1, 1)
    if nhwc:
        x, wt = x.contiguous(memory_format=torch.channels_last), wt.contiguous(memory_format=torch.channels_last)
    for L in (32, 64, 128):
        args = (L, lfsr, 16, (1, 1), (1, 1), (7, 8, 1), 1, 1, xnor, False)
        want = oracle.conv2d_generic_general_split(x, wt, *args)
        assert int(want[0].sum()) > 0
        for kernel in ("tensor", "direct"):
            ops.set_conv_kernel(kernel)
            try:
                got = ops.conv2d_generic_general_split_acc(x.cuda(), wt.cuda(), *args)
            finally:
                ops.set_conv_kernel("auto")
            assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1]), (kernel, L)


@pytest.mark.parametrize("c,k,low,co", [(2016, 1, 0.9, 64), (227, 3, 0.9, 70), (504, 2, 0.9, 64),   # every count is summed as it is
                                        (8191, 1, 0.3, 64), (910, 3, 0.3, 64), (2047, 2, 0.3, 70)])  # counts around the limit
@pytest.mark.parametrize("nhwc", [True, False])
def test_counts_in_the_thousands(ops, c, k, low, co, nhwc):
    """Dense operands, an output channel's weights of one sign, the largest n: fp32 accumulators have to hold integers
    of this size exactly on top of their 2^23."""
    g = torch.Generator(device="cuda").manual_seed(c)
    x = torch.rand(2, c, 5, 7, device="cuda", generator=g) * (1 - low) + low
    wt = torch.rand(co, c, k, k, device="cuda", generator=g) * (1 - low) + low
    wt[1::2] *= -1
    fmt = torch.channels_last if nhwc else torch.contiguous_format
    x, wt = x.contiguous(memory_format=fmt), wt.contiguous(memory_format=fmt)
    out = []
    for kernel in ("tensor", "direct"):
        ops.set_conv_kernel(kernel)
        try:
            out.append(ops.conv2d_generic_general_split_acc(x, wt, 32, -1, 16, (0, 0), (1, 1), (7, 8, 1), 2046, 1, True, False))
            assert ops.workspace_status() == 0
        finally:
            ops.set_conv_kernel("auto")
    sums = [t.to(torch.int32) & 0xffff for t in out[1]]
    assert sums[0][:, 0::2].float().mean() > 32 * 1500 and sums[1][:, 1::2].float().mean() > 32 * 1500
    for a, b in zip(*out):
        assert torch.equal(a, b), f"{(a != b).sum().item()} counts differ"


@pytest.mark.parametrize("c,co,k", [(500, 300, 3), (402, 260, 3), (1000, 1030, 1)])
@pytest.mark.parametrize("w_nhwc", [True, False])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L", [32, 64])
def test_large_filters(ops, c, co, k, w_nhwc, w_dtype, L):
    """Weights expanded in blocks of 32 output channels (512 blocks and more): channels that end inside a word, output
    channels that end inside a block, vector and scalar loads, one and two words per stream."""
    g = torch.Generator(device="cuda").manual_seed(c + co)
    x = (torch.randn(1, c, 5, 6, device="cuda", generator=g) * 0.45).clamp(0, 1)
    wt = (torch.randn(co, c, k, k, device="cuda", generator=g) * 0.2).clamp(-1, 1).to(w_dtype)
    wt[0, :, 0, 0] = float("nan")
    wt = wt.contiguous(memory_format=torch.channels_last if w_nhwc else torch.contiguous_format)
    p = k // 2
    out = []
    for kernel in ("tensor", "direct"):
        ops.set_conv_kernel(kernel)
        try:
            out.append(ops.conv2d_generic_general_split_acc(x, wt, L, -1, 16, (p, p), (1, 1), (7, 8, 1), 2, 1, True, False))
        finally:
            ops.set_conv_kernel("auto")
    for a, b in zip(*out):
        assert torch.equal(a, b), f"{(a != b).sum().item()} counts differ"


@pytest.mark.parametrize("L", [32, 64])
@pytest.mark.parametrize("c,co", [(1000, 1000), (998, 1030)])
def test_large_linear_layer_with_seeds_of_its_own(ops, L, c, co):
    """The same blocks with linear seeds, other offsets for positive than for negative weights."""
    g = torch.Generator().manual_seed(c)
    top = (L - 1) / L
    x = ((torch.rand(3, c, generator=g) * 128).floor() / 128).clamp(max=top)
    wt = ((torch.randn(co, c, generator=g) * 0.2).clamp(-1, 1) * 128).round().div(128).clamp(-top, top)
    want = _torch_loop_linear_counts(x.numpy(), wt.numpy(), L, (67, 37), True)
    got = ops.linear_generic_general_acc(x.cuda(), wt.cuda(), (7, 8, 1), L, -1, 0, 1, False, False, weight_seeds=(67, 37))
    assert all((t.cpu().numpy() == w).all() for t, w in zip(got, want))
