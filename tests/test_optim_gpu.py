"""Multi-tensor Adam kernel against torch.optim (fp32 reference of the same update)."""
import pytest
import torch

from physicsnemo_b200.optim import FusedAdam, grad_global_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wmode", [False, True])
def test_fused_adam_kernel(wmode):
    torch.manual_seed(0)
    shapes = [(256, 256), (1024,), (3, 5, 7), (1,), (8192 * 3 + 17,)]
    pa = [torch.randn(s, device="cuda") for s in shapes]
    pb = [p.clone() for p in pa]
    ours = FusedAdam(pa, lr=1e-2, weight_decay=0.05, adam_w_mode=wmode)
    ref = (torch.optim.AdamW if wmode else torch.optim.Adam)(pb, lr=1e-2, weight_decay=0.05)
    for s in range(4):
        for i, (a, b) in enumerate(zip(pa, pb)):
            torch.manual_seed(100 * s + i)
            g = torch.randn_like(a)
            a.grad, b.grad = g, g.float()
        ours.step(), ref.step()
    assert ours.kernel_launches == 4
    for a, b in zip(pa, pb):
        assert torch.allclose(a, b, atol=1e-5, rtol=1e-4)


def test_grad_norm_kernel():
    ps = [torch.nn.Parameter(torch.randn(n, device="cuda")) for n in (5, 70000, 8192)]
    for i, p in enumerate(ps):
        p.grad = torch.randn_like(p)
    ref = torch.sqrt(sum((p.grad.float() ** 2).sum() for p in ps))
    assert torch.allclose(grad_global_norm(ps), ref, rtol=1e-4)


def test_fused_adam_alternating_grad_buffers_without_sync():
    """Gradient buffers change from step to step and the host runs ahead of the device (a long kernel is queued before
    every step): each step must still read ITS pointers from the staged table."""
    torch.manual_seed(1)
    shapes = [(512, 512), (4097,), (64, 3)]
    pa = [torch.randn(s, device="cuda") for s in shapes]
    pb = [p.clone() for p in pa]
    ours = FusedAdam(pa, lr=3e-3)
    ref = torch.optim.Adam(pb, lr=3e-3)
    pool = [[torch.randn_like(p) for p in pa] for _ in range(5)]        # five distinct sets of gradient tensors
    big = torch.randn(8192, 8192, device="cuda")
    for s in range(10):
        _ = big @ big                                                   # keeps the device behind the host
        for a, b, g in zip(pa, pb, pool[s % 5]):
            a.grad, b.grad = g, g.clone()
        ours.step()
    torch.cuda.synchronize()
    for s in range(10):
        for b, g in zip(pb, pool[s % 5]):
            b.grad = g.clone()
        ref.step()
    for a, b in zip(pa, pb):
        assert torch.allclose(a, b, atol=1e-5, rtol=1e-4)


def test_fused_adam_capturable_resume_keeps_step_count():
    """A capturable optimizer's step count lives on the device and advances in graph replays; ``state_dict`` must carry
    it, and a fresh optimizer that loads it must continue with the same bias correction as torch.optim.Adam."""
    torch.manual_seed(2)
    p0 = torch.randn(1000, device="cuda")
    grads = [torch.randn(1000, device="cuda") for _ in range(8)]
    a, b = p0.clone(), p0.clone()
    ours = FusedAdam([a], lr=1e-2, capturable=True)
    ref = torch.optim.Adam([b], lr=1e-2)
    static_g = torch.zeros_like(a)
    a.grad = static_g
    static_g.copy_(grads[0])
    ours.step()                                             # warm-up step (eager)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                           # capture runs nothing: the replays below are steps 2 .. 5
        ours.step()
    for g in grads[1:5]:
        static_g.copy_(g)
        graph.replay()
    torch.cuda.synchronize()
    sd = ours.state_dict()
    assert sd["state"][0]["step"] == 5
    a2 = a.detach().clone()
    resumed = FusedAdam([a2], lr=1e-2, capturable=True)
    resumed.load_state_dict(sd)
    for g in grads[5:]:
        a2.grad = g.clone()
        resumed.step()
    for g in grads:
        b.grad = g.clone()
        ref.step()
    assert torch.allclose(a2, b, atol=1e-5, rtol=1e-4)


@pytest.mark.parametrize("width,layers", [(128, 2), (256, 1)])       # one kernel for the whole MLP; layer by layer
def test_fused_adam_step_reaches_the_next_forward(width, layers):
    """The MLPs work on bf16 copies of their matrices: a step must be seen by the next forward and by its backward."""
    from physicsnemo_b200.nn.module.gnn_layers.mesh_graph_mlp import MeshGraphMLP

    m = MeshGraphMLP(width, width, width, layers, torch.nn.SiLU()).cuda()
    opt = FusedAdam(m.parameters(), lr=5e-2)
    x = torch.randn(300, width, device="cuda").bfloat16()
    for step in range(3):
        leaf = x.clone().requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(leaf)
        opt.zero_grad()
        y.backward(x)
        twin = MeshGraphMLP(width, width, width, layers, torch.nn.SiLU()).double().cuda()
        twin.load_state_dict(m.state_dict())
        ref_leaf = x.double().requires_grad_()
        ref = twin(ref_leaf)
        ref.backward(x.double())
        # bf16 products against 64 bits; the step moves every weight by about half its spread
        assert (y.double() - ref).norm() < 1.5e-2 * ref.norm(), step
        assert (leaf.grad.double() - ref_leaf.grad).norm() < 3e-2 * ref_leaf.grad.norm(), step
        versions = [p._version for p in m.parameters()]
        opt.step()
        assert all(p._version > v for p, v in zip(m.parameters(), versions))


def test_captured_step_trains_the_matrices_it_reads():
    from physicsnemo_b200 import ops
    from physicsnemo_b200.utils.capture import GraphedStep

    w = torch.nn.Parameter(torch.randn(64, 128, device="cuda") / 128 ** 0.5)
    opt = FusedAdam([w], lr=5e-2, capturable=True)
    x = torch.randn(256, 128, device="cuda").bfloat16().requires_grad_()
    before = torch.empty_like(w)

    def step(t):
        t.grad = w.grad = None
        before.copy_(w.detach())
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = ops.linear(t, w)
        y.square().mean().backward()
        opt.step()
        return y.detach(), t.grad

    step(x)
    graphed = GraphedStep(step, [x], warmup=1)
    for k in range(3):
        y, dx = graphed()
        ref = x.detach().double() @ before.double().t()
        gref = (2 / ref.numel()) * ref @ before.double()
        assert (y.double() - ref).norm() < 1e-2 * ref.norm(), k
        assert (dx.double() - gref).norm() < 2e-2 * gref.norm(), k
        # a forward between replays: the graph changed the parameter, and its version does not say so
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            now = ops.linear(x.detach(), w)
        ref = x.detach().double() @ w.detach().double().t()
        assert (now.double() - ref).norm() < 1e-2 * ref.norm(), k


def test_captured_optimizer_step_reaches_eager_forwards():
    """The step alone in a graph, forward and backward launched from the host."""
    from physicsnemo_b200 import ops

    w = torch.nn.Parameter(torch.randn(64, 128, device="cuda") / 128 ** 0.5)
    w.grad = torch.randn_like(w)
    opt = FusedAdam([w], lr=5e-2, capturable=True)
    x = torch.randn(256, 128, device="cuda").bfloat16()

    def agrees():
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            y = ops.linear(x, w)
        ref = x.double() @ w.detach().double().t()
        return float((y.double() - ref).norm()) < 1e-2 * float(ref.norm())

    assert agrees()
    opt.step()
    assert agrees()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        opt.step()
    for _ in range(3):
        graph.replay()
        assert agrees()
