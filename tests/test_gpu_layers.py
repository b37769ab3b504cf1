"""The layer calls of the path on the GPU against the CPU checker: `QuantizedLinear`, `Expert`, `MLP` and dense
`Linear` `forward_with_stream` (mlx/src/nn/linear.rs:51-63,170-177, mlx/src/nn/moe.rs:26-32,
mlx/src/nn/mlp.rs:27-33), each one call into the C ABI."""
import numpy as np
import pytest
import torch

from ironmlx_b200 import _lib, nn
from ironmlx_b200.workloads import MoEConfig, Workload, normal, round_bf16
from oracle import formats as F
from oracle import moe as O
from gpu_util import bf16_to_np, q_to_device, t_bf16
from util import quantize_stack, squeeze0

pytestmark = pytest.mark.gpu
TOL = 2e-3


def _qlinear(out_dim, in_dim, mode, bits, group, seed):
    cfg = MoEConfig("l", 1, in_dim, 1, 1, out_dim, mode=mode, bits=bits, group_size=group, seed=seed)
    w = round_bf16(normal(seed, "w", (out_dim, in_dim), 0.02))
    return squeeze0(quantize_stack([w], cfg))


@pytest.mark.parametrize("mode,bits,group", [("affine", 4, 64), ("affine", 8, 64), ("affine", 2, 64), ("mxfp8", 8, 32),
                                             ("nvfp4", 4, 16)])
@pytest.mark.parametrize("m,in_dim,out_dim", [(1, 2048, 512), (8, 512, 2048), (40, 1024, 1024), (300, 2048, 512),
                                              (70, 512, 20480),        # a vocabulary-sized output on the tensor-core kernel
                                              (5, 192, 320)])          # the last shape: the scalar fallback
def test_quantized_linear_forward(cuda, m, in_dim, out_dim, mode, bits, group):
    if in_dim % group:
        pytest.skip("input dimension not a multiple of the group size")
    q = _qlinear(out_dim, in_dim, mode, bits, group, seed=7)
    x = round_bf16(normal(8, "x", (m, in_dim)))
    ref = F.quantized_matmul(x, q.w, q.scales, q.biases, True, group, bits, mode, global_scale=q.global_scale)
    ql = q_to_device(q, cuda)
    y = bf16_to_np(ql.forward_with_stream(t_bf16(x, cuda)))
    assert y.shape == (m, out_dim)
    assert O.rel_l2(y, ref) <= TOL


@pytest.mark.parametrize("mode,bits,group", [("affine", 4, 64), ("mxfp8", 8, 32)])
@pytest.mark.parametrize("m", [3, 70, 400])
def test_expert_and_mlp_forward(cuda, m, mode, bits, group):
    cfg = MoEConfig("e", m, 1024, 2, 1, 512, 512, mode=mode, bits=bits, group_size=group, seed=11)
    from util import make_params
    x, p = make_params(cfg)
    from gpu_util import moe_to_device
    moe = moe_to_device(p, cuda)
    xd = t_bf16(x, cuda)
    # a routed expert: views into the fused tensors (gate and up rows adjacent)
    e1 = moe._fused.expert(1)
    wg, wu, wd = O.expert_weights(p, 1)
    ref = O.swiglu_mlp(x, wg, wu, wd)
    y = bf16_to_np(e1.forward_with_stream(xd))
    assert O.rel_l2(y, ref) <= TOL
    # the shared expert: three separate tensors
    sg = F.dequantize(p.shared_gate_proj.w, p.shared_gate_proj.scales, p.shared_gate_proj.biases, group, bits, mode,
                      p.shared_gate_proj.global_scale)
    su = F.dequantize(p.shared_up_proj.w, p.shared_up_proj.scales, p.shared_up_proj.biases, group, bits, mode,
                      p.shared_up_proj.global_scale)
    sd = F.dequantize(p.shared_down_proj.w, p.shared_down_proj.scales, p.shared_down_proj.biases, group, bits, mode,
                      p.shared_down_proj.global_scale)
    ref_s = O.swiglu_mlp(x, sg, su, sd)
    ys = bf16_to_np(moe.shared_expert.forward_with_stream(xd))
    assert O.rel_l2(ys, ref_s) <= TOL


@pytest.mark.parametrize("m,in_dim,out_dim,bias", [(1, 2048, 256, False), (70, 512, 1, False), (130, 256, 100, True)])
def test_dense_linear_forward(cuda, m, in_dim, out_dim, bias):
    w = round_bf16(normal(3, "w", (out_dim, in_dim), 0.05))
    b = round_bf16(normal(3, "b", (out_dim,), 0.1)) if bias else None
    x = round_bf16(normal(4, "x", (m, in_dim)))
    ref = x.astype(np.float64) @ w.astype(np.float64).T + (0 if b is None else b.astype(np.float64))
    lin = nn.Linear(t_bf16(w, cuda), None if b is None else t_bf16(b, cuda))
    y = bf16_to_np(lin.forward_with_stream(t_bf16(x, cuda)))
    assert y.shape == (m, out_dim)
    assert O.rel_l2(y, ref) <= TOL
    assert np.abs(y - ref).max() <= 2.0 ** -7 * np.abs(ref).max() + 1e-6


def test_fusing_experts_with_different_tensor_scales_is_refused(cuda):
    q = _qlinear(128, 128, "nvfp4", 4, 16, seed=2)
    a = q_to_device(q, cuda)
    b = q_to_device(q, cuda)
    b.global_scale = (a.global_scale or 1.0) * 2
    with pytest.raises(_lib.IronMLXError):
        nn.FusedExperts.from_experts([nn.Expert(a, a, a), nn.Expert(b, b, b)])


@pytest.mark.parametrize("mode,bits,group,m", [("affine", 4, 64, 40), ("affine", 4, 64, 3), ("affine", 8, 64, 3), ("nvfp4", 4, 16, 3),
                                               ("mxfp8", 8, 32, 200), ("affine", 6, 64, 40), ("affine", 4, 64, 5)])
@pytest.mark.parametrize("at", [1, 2, 4])
def test_quantized_linear_into_rows_at_any_value(cuda, mode, bits, group, m, at):
    """`imx_quantized_matmul_ws` with y at 2, 4 and 8 bytes past a multiple of 16: the values of the aligned call (the
    4-bit decode kernel that takes odd addresses adds in another order: one step of bf16), nothing around them."""
    import ctypes as C
    n_in, n_out = (512, 384) if m == 5 else (512, 1024)
    ql = q_to_device(_qlinear(n_out, n_in, mode, bits, group, seed=17), cuda)
    x = t_bf16(round_bf16(normal(18, "x", (m, n_in))), cuda)
    want = ql.forward_with_stream(x)
    buf = torch.full((m * n_out + 16,), 7.0, dtype=torch.bfloat16, device=cuda)
    nb, qt, lib = C.c_size_t(0), ql.qtensor(), _lib.lib()
    fmt = (group, bits, _lib.MODE[mode])
    _lib.check(lib.imx_quantized_matmul_scratch_bytes(m, n_out, n_in, *fmt, C.byref(nb)))
    scratch = torch.zeros(nb.value, dtype=torch.uint8, device=cuda)
    _lib.check(lib.imx_quantized_matmul_ws(x.data_ptr(), m, C.byref(qt), n_out, n_in, *fmt, buf.data_ptr() + 2 * at,
                                           scratch.data_ptr(), nb.value, torch.cuda.current_stream().cuda_stream))
    got = buf[at:at + m * n_out].view(m, n_out)
    assert (buf[:at] == 7).all() and (buf[at + m * n_out:] == 7).all()
    if (mode, bits, m, at) == ("affine", 4, 3, 1):
        assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 1e-6).all()
    else:
        assert torch.equal(got, want)
    assert lib.imx_quantized_matmul_ws(x.data_ptr(), m, C.byref(qt), n_out, n_in, *fmt, buf.data_ptr() + 1,
                                       scratch.data_ptr(), nb.value, torch.cuda.current_stream().cuda_stream) == _lib.ERR_INVALID


@pytest.mark.parametrize("mode,bits,group,m", [("affine", 6, 64, 3), ("affine", 3, 64, 70), ("mxfp8", 8, 32, 12)])
def test_expert_rows_beyond_the_range_of_fp16(cuda, mode, bits, group, m):
    """The fp16 copy of an expert's input is clamped to +-65504, as in the block: the outputs are those of the clamped
    rows (fp16 carries them exactly), and rows beside them are not touched."""
    from gpu_util import moe_to_device
    from util import make_params
    cfg = MoEConfig("range", m, 1024, 1, 1, 512, 0, mode=mode, bits=bits, group_size=group, seed=31)
    x, p = make_params(cfg)
    expert = moe_to_device(p, cuda)._fused.expert(0)
    xd = t_bf16(x, cuda)
    clean = expert.forward_with_stream(xd)
    xd[1, 7], xd[1, 100] = 1e5, -float("inf")
    y = expert.forward_with_stream(xd)
    clamped = bf16_to_np(xd[1:2]).clip(-65504.0, 65504.0).astype(np.float64)
    wg, wu, wd = (w.astype(np.float64) for w in O.expert_weights(p, 0))
    with np.errstate(over="ignore"):
        act = np.clip(O.silu(clamped @ wg.T) * (clamped @ wu.T), -65504.0, 65504.0)
    assert O.rel_l2(bf16_to_np(y[1:2]), act @ wd.T) <= TOL
    rest = torch.arange(m, device=cuda) != 1
    assert torch.equal(y[rest], clean[rest])
