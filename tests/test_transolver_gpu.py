"""Fused sm_100a Transolver path against the plain PyTorch fp32 path of the same model."""
import copy

import pytest
import torch

from physicsnemo_b200 import ops
from physicsnemo_b200.models.transolver import Transolver

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


def test_fused_block_matches_fp32_reference():
    dev = torch.device("cuda")
    model = Transolver(functional_dim=3, out_dim=4, embedding_dim=3, n_layers=2, n_hidden=256, n_head=8,
                       slice_num=64, mlp_ratio=4, use_te=False).to(dev)
    # move away from the init point so every parameter matters
    with torch.no_grad():
        for p in model.parameters():
            p.add_(torch.randn_like(p) * 0.02)
    ref = copy.deepcopy(model)
    n = 5000
    fx, emb = torch.randn(1, n, 3, device=dev), torch.randn(1, n, 3, device=dev)
    tgt = torch.randn(1, n, 4, device=dev)
    before = ops.kernel_launches()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        out = model(fx, embedding=emb)
    loss = torch.nn.functional.mse_loss(out.float(), tgt)
    loss.backward()
    assert ops.kernel_launches() - before >= 20, "fused kernels were not used"
    out_ref = ref(fx, embedding=emb)  # fp32, PyTorch ops only
    loss_ref = torch.nn.functional.mse_loss(out_ref, tgt)
    loss_ref.backward()
    assert ops.device_error() == 0
    assert _rel(out, out_ref) < 3e-2, _rel(out, out_ref)
    # every gradient within 2 % of its own norm plus 1 % of the model's total gradient norm (the floor covers tensors
    # whose gradient nearly cancels at this point, e.g. the slice projections: they move by a few % of their own tiny
    # norm between two runs of the same bf16 model)
    total = torch.sqrt(sum(q.grad.float().pow(2).sum() for q in ref.parameters())).item()
    bad = []
    for (name, p), (_, q) in zip(model.named_parameters(), ref.named_parameters()):
        assert p.grad is not None, name
        d = (p.grad.float() - q.grad.float()).norm().item()
        r = d / (q.grad.float().norm().item() + 1e-2 * total)
        if r > 2e-2:
            bad.append((name, r))
    assert not bad, bad


def test_fused_batch_two():
    dev = torch.device("cuda")
    model = Transolver(functional_dim=2, out_dim=1, embedding_dim=3, n_layers=1, n_hidden=128, n_head=4,
                       slice_num=64, use_te=False).to(dev)
    ref = copy.deepcopy(model)
    fx, emb = torch.randn(2, 777, 2, device=dev), torch.randn(2, 777, 3, device=dev)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        out = model(fx, embedding=emb)
    assert _rel(out, ref(fx, embedding=emb)) < 3e-2


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,cout", [(8, 32, 256), (8, 32, 264), (3, 16, 72), (4, 8, 200), (2, 4, 64), (3, 2, 40), (1, 1, 8), (8, 64, 512), (2, 64, 264),
                                      (1, 64, 64)])
def test_slice_token_kernels(H, D, cout):
    """Slice-token attention and its backward, head widths below and at the tile, one to five chunks of 64 output channels (a head has at
    most four CTAs), against autograd in 64 bits.  fp32 sums of at most 512 terms; bf16 results carry 2^-9 of a value."""
    from physicsnemo_b200.ops import pa_small as P

    S, g = P.S, torch.Generator(device="cuda").manual_seed(H * D + cout)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    sums, norm = rn(H * S, H * D) * 20, 5 + 10 * torch.rand(H * S, generator=g, device="cuda")
    Wqkv, Wo, dwc = rn(3 * D, D) / D ** 0.5, rn(cout, H * D) / (H * D) ** 0.5, rn(cout, H * S)
    buf = torch.cat((sums.reshape(-1), norm))
    wcomb16, saved = P.tokens_fwd([buf.data_ptr()], sums.numel(), H * D, Wqkv, Wo, H, D)
    dWo, dWqkv, d_norm, Bcat, BdT = P.tokens_bwd([dwc.data_ptr()], Wqkv, Wo, saved, H, D, 0.5)

    eye = torch.eye(H, device="cuda", dtype=torch.float64)
    raw = torch.stack([sums[h * S:(h + 1) * S, h * D:(h + 1) * D] for h in range(H)]).double().requires_grad_(True)
    nrm, wq, wo = (t.double().requires_grad_(True) for t in (norm.reshape(H, S), Wqkv, Wo))
    tok = raw / (nrm + 1e-2)[..., None]
    q, k, v = (tok @ wq.t()).chunk(3, -1)
    out = torch.softmax(q @ k.transpose(1, 2) * D ** -0.5, -1) @ v
    wcomb = torch.einsum("chd,hsd->chs", wo.reshape(cout, H, D), out).reshape(cout, H * S)
    draw, dn, dwq, dwo = torch.autograd.grad(wcomb, (raw, nrm, wq, wo), dwc.double())

    def close(a, b, tol):
        assert float((a.double() - b).norm() / b.norm()) < tol

    close(P.saved_parts(saved, H, D, cout)[7], wcomb, 1e-5)
    close(wcomb16, wcomb, 2.0 ** -8)
    close(dWo, 0.5 * dwo, 1e-5)
    close(dWqkv, 0.5 * dwq, 1e-5)
    close(d_norm, dn.reshape(-1), 1e-4)                                  # a sum that partly cancels
    blocks = torch.einsum("hsd,hg->hsgd", draw, eye).reshape(H * S, H * D)
    close(Bcat, torch.cat((wcomb.t(), blocks), 1), 2.0 ** -8)
    close(BdT, blocks.t(), 2.0 ** -8)
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dim,heads,dim_head", [(256, 8, 64), (128, 1, 64), (72, 4, 16), (200, 8, 32)])
def test_training_call_of_the_module(dim, heads, dim_head):
    """Whatever the fused path takes forward it takes backward: the module's default head width, widths that are no multiple of 64, against
    the plain path in fp32.  Gradients are compared as in the test of a block."""
    from physicsnemo_b200.nn.module.physics_attention import PhysicsAttentionIrregularMesh

    torch.manual_seed(dim)
    mod = PhysicsAttentionIrregularMesh(dim, heads=heads, dim_head=dim_head, slice_num=64, use_te=False).cuda()
    with torch.no_grad():
        for p in mod.parameters():
            p.add_(torch.randn_like(p) * 0.02)
    ref = copy.deepcopy(mod)
    x = torch.randn(1, 3001, dim, device="cuda")
    g = torch.randn_like(x)
    xs = [x.clone().requires_grad_(True) for _ in range(2)]
    before = ops.kernel_launches()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        out = mod(xs[0])
    out.float().backward(g)
    assert ops.kernel_launches() - before >= 10, "fused kernels were not used"
    want = ref(xs[1])
    want.backward(g)
    assert ops.device_error() == 0
    assert _rel(out, want) < 3e-2
    assert _rel(xs[0].grad, xs[1].grad) < 3e-2
    total = torch.sqrt(sum(q.grad.float().pow(2).sum() for q in ref.parameters())).item()
    for (name, p), (_, q) in zip(mod.named_parameters(), ref.named_parameters()):
        assert (p.grad.float() - q.grad.float()).norm().item() < 2e-2 * (q.grad.float().norm().item() + 1e-2 * total), name
        assert p.grad.untyped_storage().nbytes() == p.grad.nbytes, name          # a buffer of its own: held and saved alone


@pytest.mark.gpu
def test_temperatures_at_the_ends_of_their_range_have_gradients():
    """The initial temperature is the lower end of the clamp, where torch passes the gradient on."""
    from physicsnemo_b200.ops import pa_small as P

    temp = torch.tensor([0.4, 0.5, 0.7, 5.0, 5.1], device="cuda")
    H, D, C = temp.numel(), 8, 64
    rn = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    sums = rn(H)                                                         # of d(logit / T) logit / T
    dtemp = P.prepare_bwd(rn(H * (P.S + D), C), rn(H * (P.S + D)), sums, rn(H * D, C), rn(H * D), rn(P.S, D), temp, H, D)[-1]
    t = temp.double().requires_grad_(True)
    (want,) = torch.autograd.grad((-sums.double() * torch.log(torch.clamp(t, min=0.5, max=5))).sum(), t)
    assert torch.allclose(dtemp.double(), want, rtol=1e-6, atol=0)
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["in_project_x", "in_project_fx", "qkv_project", "out_linear"])
def test_parameters_that_lie_by_columns(name):
    """A weight given as a transposed view is the same weight: the kernels, which read parameters as they lie, leave it to the plain path."""
    from physicsnemo_b200.nn.module.physics_attention import PhysicsAttentionIrregularMesh

    torch.manual_seed(7)
    mod = PhysicsAttentionIrregularMesh(64, heads=2, dim_head=32, slice_num=64, use_te=False).cuda()
    x = torch.randn(1, 500, 64, device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        want = mod(x)
        layer = getattr(mod, name)
        layer.weight = torch.nn.Parameter(layer.weight.t().contiguous().t())
        assert not layer.weight.is_contiguous()
        assert _rel(mod(x), want) < 2e-2
    assert ops.device_error() == 0
