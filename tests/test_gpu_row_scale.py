"""A factor per row on the tensor-core expert kernels (`imx_moe_experts`): it is the row's own, whatever factor the
format keeps per weight row."""
import pytest
import torch

from ironmlx_b200.ep import CudaStages
from ironmlx_b200.workloads import MoEConfig
from gpu_util import moe_to_device, t_bf16
from util import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,bits,group", [("mxfp8", 8, 32), ("nvfp4", 4, 16), ("affine", 4, 64)])
def test_row_scale_of_the_expert_stage(cuda, mode, bits, group):
    """`imx_moe_experts` with a factor per row on the tensor-core kernels: the factor times the unscaled rows (two
    fp32 roundings)."""
    cfg = MoEConfig("scaled", tokens=80, hidden=512, num_experts=2, top_k=1, intermediate=512, mode=mode, bits=bits,
                    group_size=group, seed=4)
    x, p = make_params(cfg)
    moe = moe_to_device(p, cuda, "prefill")
    c = moe.config()
    x16 = t_bf16(x, cuda).to(torch.float16)
    off = torch.tensor([0, 50, 80], dtype=torch.int32, device=cuda)
    scale = torch.linspace(0.1, 3.0, 80, device=cuda)
    st = CudaStages(cuda)
    plain = st.experts(c, moe._fused.gate_up, moe._fused.down, 2, x16, None, off, 80, None).clone()
    scaled = st.experts(c, moe._fused.gate_up, moe._fused.down, 2, x16, None, off, 80, scale)
    want = plain.double() * scale.double()[:, None]
    assert ((scaled.double() - want).abs() <= 2.0 ** -22 * want.abs()).all()
