"""The tensor-core kernels with two-term weights (affine 3/5/6-bit, 4-bit in groups of 32): the formats whose
weights stay in 32 bits, against fp64 and against the scalar kernels they replace."""
import ctypes as C

import numpy as np
import pytest
import torch

from ironmlx_b200 import _lib, nn, ops
from ironmlx_b200.workloads import MoEConfig
from oracle import moe as O
from gpu_util import bf16_to_np, moe_to_device, t_bf16
from util import make_params

pytestmark = pytest.mark.gpu

FORMATS = [(3, 64), (5, 64), (6, 64), (4, 32), (6, 32), (3, 128)]


def _layer(cuda, n_out, n_in, bits, group, seed, scale=0.02):
    gen = torch.Generator(device=cuda)
    gen.manual_seed(seed)
    w = torch.randn(n_out, n_in, generator=gen, device=cuda) * scale
    q = ops.quantize(w, group, bits)
    wd = ops.dequantize(*q, group, bits, dtype=torch.float32).double()
    return nn.QuantizedLinear(*q, group, bits), wd, gen


def _check(y, x, wd, in_dim):
    """One rounding to bf16 (half a unit in the last of 8 bits: 2^-8 of the value at most), 2^-22 per weight (two fp16
    terms) and the fp32 sums: at most n + 2 roundings of 2^-24 each of the sum of magnitudes."""
    xd = x.double()
    ref = xd @ wd.T
    mags = xd.abs() @ wd.abs().T
    bound = 2.0 ** -8 * ref.abs() + (2.0 ** -22 + (in_dim + 2) * 2.0 ** -24) * mags
    assert torch.isfinite(y).all()
    assert ((y.double() - ref).abs() <= bound).all(), ((y.double() - ref).abs() / bound).max().item()


@pytest.mark.parametrize("bits,group", FORMATS)
@pytest.mark.parametrize("m,in_dim,out_dim", [(1, 2048, 512), (17, 1024, 128), (129, 512, 384), (257, 1024, 256)])
def test_linear(cuda, bits, group, m, in_dim, out_dim):
    layer, wd, gen = _layer(cuda, out_dim, in_dim, bits, group, 3)
    x = torch.randn(m, in_dim, generator=gen, device=cuda)
    # differences of two weights of a group: what a weight rounded to 16 bits gets wrong
    if m > 8:
        x[1::2] = 0
        i = torch.randint(0, in_dim // group, (x[1::2].shape[0],), generator=gen, device=cuda) * group
        r = torch.arange(x[1::2].shape[0], device=cuda) * 2 + 1
        x[r, i + torch.randint(0, group // 2, i.shape, generator=gen, device=cuda)] = 1.0
        x[r, i + group // 2 + torch.randint(0, group // 2, i.shape, generator=gen, device=cuda)] = -1.0
    x = x.to(torch.bfloat16)
    _check(layer.forward_with_stream(x), x, wd, in_dim)


@pytest.mark.parametrize("bits,group", FORMATS)
@pytest.mark.parametrize("m,in_dim,out_dim", [(6, 2048, 2048), (200, 2048, 512)])
def test_linear_error_is_that_of_the_scalar_kernel(cuda, bits, group, m, in_dim, out_dim):
    """Against fp64 in the 2-norm: the rounding to bf16 leaves 1.66e-3 on either, what the two terms and the tensor cores'
    sums add is a few 1e-6 of the value (1e-5 of that error; 1e-4 allowed)."""
    layer, wd, gen = _layer(cuda, out_dim, in_dim, bits, group, 19)
    x = torch.randn(m, in_dim, generator=gen, device=cuda).to(torch.bfloat16)
    ref = x.double() @ wd.T
    y, z, qt = layer.forward_with_stream(x), torch.empty(m, out_dim, dtype=torch.bfloat16, device=cuda), layer.qtensor()
    _lib.check(_lib.lib().imx_quantized_matmul(x.data_ptr(), m, C.byref(qt), out_dim, in_dim, 1, group, bits, 0, z.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream))
    assert (y.double() - ref).norm() <= (1 + 1e-4) * (z.double() - ref).norm()


@pytest.mark.parametrize("bits,group,in_dim", [(6, 64, 9728), (6, 64, 11008), (3, 64, 8192), (5, 32, 5120), (6, 32, 4096)])
@pytest.mark.parametrize("m,out_dim", [(3, 384), (20, 512)])
def test_linear_of_long_rows(cuda, bits, group, in_dim, m, out_dim):
    """Rows of scales that leave little shared memory beside them, with weight tiles that pair up (512) and do not (384)."""
    layer, wd, gen = _layer(cuda, out_dim, in_dim, bits, group, 11)
    x = torch.randn(m, in_dim, generator=gen, device=cuda).to(torch.bfloat16)
    _check(layer.forward_with_stream(x), x, wd, in_dim)


@pytest.mark.parametrize("bits,group", [(6, 64), (3, 64)])
@pytest.mark.parametrize("x_scale,w_scale", [(1e20, 1e-12), (1e-25, 1e10), (1e-3, 1e-6), (70000.0, 3.0)])
def test_linear_outside_the_range_of_fp16(cuda, bits, group, x_scale, w_scale):
    layer, wd, gen = _layer(cuda, 256, 512, bits, group, 5, w_scale)
    x = (torch.randn(40, 512, generator=gen, device=cuda) * x_scale)
    x[3] = 0
    x[4] *= 1e-6
    x = x.to(torch.bfloat16)
    _check(layer.forward_with_stream(x), x, wd, 512)


@pytest.mark.parametrize("bits,group,m", [(6, 64, 40), (3, 128, 3), (5, 64, 300), (6, 32, 17)])
def test_linear_rows_with_infinities(cuda, bits, group, m):
    """Rows with infinities or NaNs come out as the scalar kernel gives them, and leave their neighbours alone."""
    layer, wd, gen = _layer(cuda, 256, 1024, bits, group, 15)
    x = torch.randn(m, 1024, generator=gen, device=cuda).to(torch.bfloat16)
    clean = layer.forward_with_stream(x)
    inf = float("inf")
    bad = x.clone()
    bad[0, 5] = inf
    bad[1, 700] = -inf
    bad[1, 1023] = -inf
    bad[1, 2] = 3e38
    if m > 3:
        bad[m - 1, ::7] = inf
        bad[4, 9], bad[4, 10] = inf, -inf
        bad[6, 100], bad[6, 101] = inf, float("nan")
    y = layer.forward_with_stream(bad)
    want = torch.empty_like(y)
    qt = layer.qtensor()
    _lib.check(_lib.lib().imx_quantized_matmul(bad.data_ptr(), m, C.byref(qt), 256, 1024, 1, group, bits, 0, want.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream))
    rows = (~torch.isfinite(bad).all(-1)).nonzero()[:, 0]
    assert torch.isinf(want[0]).any() and torch.equal(torch.nan_to_num(y[rows], nan=5.0), torch.nan_to_num(want[rows], nan=5.0))
    fine = torch.isfinite(bad).all(-1)
    assert torch.equal(y[fine], clean[fine])


@pytest.mark.parametrize("bits,group", FORMATS)
@pytest.mark.parametrize("tokens,experts,top_k,shared", [(1, 8, 2, 512), (70, 4, 2, 0), (300, 3, 2, 512)])
def test_block(cuda, bits, group, tokens, experts, top_k, shared):
    cfg = MoEConfig("two-term", tokens=tokens, hidden=1024, num_experts=experts, top_k=top_k, intermediate=512,
                    shared_intermediate=shared, bits=bits, group_size=group, seed=9)
    x, p = make_params(cfg)
    moe = moe_to_device(p, cuda)
    xd = t_bf16(x, cuda)
    a = bf16_to_np(moe.forward_with_stream(xd))
    moe.check_status()
    b = bf16_to_np(moe.forward_with_stream(xd, path="generic"))
    ref = O.moe_forward(x, p).y
    assert O.rel_l2(a, ref) <= 2e-3
    # no further from the checker than the scalar kernels (2 %: values that fall on either side of a rounding)
    assert O.rel_l2(a, ref) <= 1.02 * O.rel_l2(b, ref)
    # both round the SwiGLU rows to fp16 and the result to bf16: single values differ by a step of each at most
    assert np.abs(a - b).max() <= 2.0 ** -8 * np.abs(b).max() * 1.5
