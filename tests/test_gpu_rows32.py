"""The tensor-core kernels where they take over from the decode kernels with the rows kept in fp32: batches between
decode and prefill sizes, and reductions whose rows of scales are not whole 16-byte pieces."""
import numpy as np
import pytest

from ironmlx_b200.workloads import MoEConfig
from oracle import moe as O
from gpu_util import bf16_to_np, moe_to_device, t_bf16
from util import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,bits,group", [("affine", 2, 64), ("affine", 4, 64), ("affine", 8, 64), ("affine", 4, 128),
                                             ("mxfp8", 8, 32), ("nvfp4", 4, 16)])
@pytest.mark.parametrize("tokens,hidden,experts,top_k,inter,shared", [
    (257, 512, 4, 2, 256, 0),         # 256-long reduction: 8 (4) bytes of scales a row; 128 rows an expert
    (260, 512, 4, 3, 256, 256),       # the same with a shared expert of several units
    (56, 1024, 4, 2, 512, 512),       # 28 rows an expert
])
def test_block_against_the_decode_kernels(cuda, mode, bits, group, tokens, hidden, experts, top_k, inter, shared):
    cfg = MoEConfig("rows32", tokens=tokens, hidden=hidden, num_experts=experts, top_k=top_k, intermediate=inter,
                    shared_intermediate=shared, mode=mode, bits=bits, group_size=group, seed=13)
    x, p = make_params(cfg)
    moe = moe_to_device(p, cuda)
    xd = t_bf16(x, cuda)
    a = bf16_to_np(moe.forward_with_stream(xd))
    moe.check_status()
    assert moe.saturations() == 0
    b = bf16_to_np(moe.forward_with_stream(xd, path="decode"))
    ref = O.moe_forward(x, p).y
    assert O.rel_l2(a, ref) <= 2e-3
    # no further from the checker than the decode kernels (2 %: values that fall on either side of a rounding)
    assert O.rel_l2(a, ref) <= 1.02 * O.rel_l2(b, ref)
    # both round the SwiGLU rows to fp16 (sums in another order: a step of 2^-10 of a few of the values that are summed)
    # and the result to bf16 (one step is 2^-7 of the value at most): single values differ by a step of bf16 and a little
    assert np.abs(a - b).max() <= (2.0 ** -7 + 2.0 ** -10) * np.abs(b).max()


@pytest.mark.parametrize("mode,bits,group,tokens,hidden,experts,top_k,inter", [
    ("nvfp4", 4, 16, 90, 512, 16, 4, 256),       # few weight tiles for an SM: 22 rows an expert
    ("mxfp8", 8, 32, 200, 512, 16, 4, 256),      # 50 rows
    ("nvfp4", 4, 16, 288, 1024, 64, 4, 512),     # a few tiles for an SM: 18 rows
    ("affine", 8, 64, 288, 1024, 64, 4, 512),
    ("affine", 4, 128, 352, 1024, 64, 4, 512),   # 22 rows
])
def test_layers_of_few_weight_tiles_stay_on_the_decode_kernels(cuda, mode, bits, group, tokens, hidden, experts, top_k, inter):
    """Where the weight tiles do not occupy the GPU the decode kernels are the faster ones up to more rows an expert: the
    call answers with their bits."""
    cfg = MoEConfig("few", tokens=tokens, hidden=hidden, num_experts=experts, top_k=top_k, intermediate=inter,
                    shared_intermediate=0, mode=mode, bits=bits, group_size=group, seed=14)
    x, p = make_params(cfg)
    moe = moe_to_device(p, cuda)
    xd = t_bf16(x, cuda)
    a, b = (bf16_to_np(moe.forward_with_stream(xd, path=path)) for path in ("auto", "decode"))
    assert np.array_equal(a, b)
