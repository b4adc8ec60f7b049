"""Edges of the tensor-core FXP conv: products that fill a slab of 128 exactly, leave a remainder or need only one;
pixels around a tile of 128; chunks of 128 output channels.  Integer work: equal to the CUDA-core kernel, which the
oracle tests cover."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,co,k,pad", [
    (1, 1, 1, 1, 1, 1, 0), (1, 16, 8, 16, 8, 1, 0), (2, 128, 8, 8, 16, 1, 0), (1, 129, 8, 16, 33, 1, 0),
    (3, 3, 11, 13, 32, 5, 2), (1, 8, 9, 9, 130, 4, 0), (2, 17, 10, 7, 64, 3, 1), (5, 64, 4, 4, 10, 4, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_tensor_kernel_equals_cuda_kernel(ops, n, c, h, w, co, k, pad, dtype):
    g = torch.Generator(device="cuda").manual_seed(c * 100 + co)
    x = torch.rand(n, c, h, w, device="cuda", generator=g).to(dtype)
    wt = (torch.randn(co, c, k, k, device="cuda", generator=g) * 0.2).clamp(-1, 1)
    out = {}
    for kernel in ("tensor", "tensor_unswizzled", "cuda"):
        ops.set_fxp_kernel(kernel)
        try:
            out[kernel] = ops.conv2d_saturate_acc(x, wt, 0, 5, 24, (pad, pad), (1, 1))
        finally:
            ops.set_fxp_kernel("auto")
    assert torch.equal(out["tensor"], out["cuda"]) and torch.equal(out["tensor_unswizzled"], out["cuda"])


@pytest.mark.parametrize("c,k", [(4, 1), (16, 1), (17, 1), (33, 1), (59, 1), (64, 1), (65, 1), (128, 1), (130, 1), (160, 1),
                                 (176, 1), (15, 3), (33, 3), (50, 2)])
@pytest.mark.parametrize("n,h,w,co", [(3, 9, 12, 10), (3, 9, 12, 83), (3, 9, 12, 300),
                                      (19, 32, 32, 10), (19, 32, 32, 300)])
def test_blocks_of_a_last_slab(ops, n, h, w, co, c, k):
    """One step and several; last slabs of one, two, three and four blocks of 32 products; one to three channel chunks;
    fewer CTAs than SMs (two weight buffers) and more (one)."""
    g = torch.Generator(device="cuda").manual_seed(c * 1000 + co)
    x = torch.rand(n, c, h, w, device="cuda", generator=g)
    wt = (torch.randn(co, c, k, k, device="cuda", generator=g) * 0.2).clamp(-1, 1)
    out = {}
    for kernel in ("tensor", "tensor_unswizzled", "cuda"):
        ops.set_fxp_kernel(kernel)
        try:
            out[kernel] = ops.conv2d_saturate_acc(x, wt, 0, 7, 24, (k // 2, k // 2), (1, 1))
            assert ops.workspace_status() == 0
        finally:
            ops.set_fxp_kernel("auto")
    assert torch.equal(out["tensor"], out["cuda"]) and torch.equal(out["tensor_unswizzled"], out["cuda"])
