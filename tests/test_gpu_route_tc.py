"""The router of larger batches (tcgen05, tiles of 32, 64 and 128 tokens) against fp64."""
import pytest
import torch

from ironmlx_b200.ep import CudaStages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,experts,hidden,k,shared,norm,bias", [
    (545, 16, 512, 4, False, True, False),      # one accumulator, a single token in the last tile
    (300, 72, 192, 8, True, False, True),       # experts that are no multiple of 32, three K steps
    (1031, 128, 1024, 4, True, True, False),    # the largest single accumulator
    (1024, 160, 64, 6, True, True, True),       # two, the second one short; one K step
    (4737, 256, 256, 8, True, True, False),     # tiles of 64
    (9473, 256, 128, 8, True, True, True),      # tiles of 128
])
def test_route(cuda, n, experts, hidden, k, shared, norm, bias):
    gen = torch.Generator(device=cuda)
    gen.manual_seed(n)
    x = torch.randn(n, hidden, generator=gen, device=cuda).to(torch.bfloat16)
    w = (torch.randn(experts, hidden, generator=gen, device=cuda) * 0.1).to(torch.bfloat16)
    sg = (torch.randn(1, hidden, generator=gen, device=cuda) * 0.1).to(torch.bfloat16) if shared else None
    b = torch.randn(experts, generator=gen, device=cuda) if bias else None
    idx, wt, gate, x16 = CudaStages(cuda).route(x, w, b, k, norm, sg)
    logits = x.double() @ w.double().T + (0 if b is None else b.double())
    p = torch.softmax(logits, -1)
    order = torch.argsort(-p, dim=-1, stable=True)
    # rows whose first k + 1 values are further apart than fp32 sums of `hidden` products can move them
    # (hidden + 1 roundings of 2^-24 of the sum of magnitudes, on either side)
    eps = 2 * (hidden + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T).amax(-1)
    top = logits.gather(1, order[:, :min(k + 1, experts)])
    clear = (top[:, :-1] - top[:, 1:] > eps[:, None]).all(-1)
    assert clear.float().mean() > 0.9
    assert torch.equal(idx[clear].long(), order[clear][:, :k])
    want = p.gather(1, order[:, :k])
    if norm:
        want = want / want.sum(-1, keepdim=True)
    # an error of eps in a logit is a factor of 1 + eps in a probability, twice with the sum; fp32 exp and quotients
    assert ((wt.double() - want).abs()[clear] <= (2 * eps[:, None] + 2.0 ** -20)[clear] * want[clear]).all()
    assert torch.equal(x16, x.to(torch.float16))
    if shared:
        z = x.double() @ sg.double().T
        assert ((gate.double() - torch.sigmoid(z)[:, 0]).abs() <= eps + 2.0 ** -20).all()


@pytest.mark.parametrize("n,experts,hidden", [(300, 16, 512), (400, 60, 2048), (900, 8, 2048)])
def test_few_tokens_and_experts_stay_on_the_kernel_per_token(cuda, n, experts, hidden):
    """Batches that would be a few tiles of the tensor-core router run on the kernel that takes a cluster per token, as
    batches below 256 tokens do: the same sums in the same order, hence the same bits for the same token."""
    gen = torch.Generator(device=cuda)
    gen.manual_seed(n)
    x = torch.randn(n, hidden, generator=gen, device=cuda).to(torch.bfloat16)
    w = (torch.randn(experts, hidden, generator=gen, device=cuda) * 0.1).to(torch.bfloat16)
    st = CudaStages(cuda)
    idx, wt = (t.clone() for t in st.route(x, w, None, 4, True, None)[:2])
    small = st.route(x[:255].contiguous(), w, None, 4, True, None)
    assert torch.equal(idx[:255], small[0]) and torch.equal(wt[:255], small[1])
