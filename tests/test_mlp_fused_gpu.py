"""The one-kernel message-passing MLP (``ops.mlp_fused``) against plain torch in 64 bits."""
import pytest
import torch
import torch.nn.functional as F

W = 128
ACTS = {1: F.gelu, 2: F.silu, 3: F.relu}


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,nodes,nsrc,act", [(1, 3, 3, 2), (127, 5, 3, 3), (128, 40, 2, 2), (129, 1, 3, 2), (148 * 128 + 1, 2000, 3, 1),
                                                 (2 * 148 * 128 + 77, 999, 1, 3), (60001, 10007, 3, 2)])
def test_mlp3_ln_forward_backward(rows, nodes, nsrc, act):
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    g = torch.Generator().manual_seed(rows + act)
    rn = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    edge, node = rn(rows, W).bfloat16(), rn(nodes, W).bfloat16()
    idx = [torch.randint(0, nodes, (rows,), generator=g) for _ in range(2)]      # nodes without a row and repeated ones occur
    params = [rn(W, W * nsrc) / (W * nsrc) ** 0.5, rn(W, W) / W ** 0.5, rn(W, W) / W ** 0.5, *(0.1 * rn(W) for _ in range(3)),
              1 + 0.1 * rn(W), 0.1 * rn(W)]
    up = rn(rows, W).bfloat16()

    leaves = [t.double().requires_grad_() for t in (edge, node, *params)]
    e, v, w1, w2, w3, b1, b2, b3, ga, be = leaves
    x = torch.cat([e, v[idx[0]], v[idx[1]]][:nsrc], 1)
    h = ACTS[act](F.linear(ACTS[act](F.linear(x, w1, b1)), w2, b2))
    ref = F.layer_norm(F.linear(h, w3, b3), (W,), ga, be) + e
    ref.backward(up.double())

    dev = [t.cuda().requires_grad_() for t in (edge, node, *params)]
    e, v, *p = dev
    segs = [None] + [ops.SegmentIndex(i.cuda(), nodes) for i in idx]
    srcs, segs = [e, v, v][:nsrc], segs[:nsrc]
    assert mf.supported(srcs, segs, p[:3], p[3:6], [act, act, 0], p[6], p[7], 0)
    out = mf.mlp3_ln(srcs, segs, p[:3], p[3:6], act, p[6], p[7], 1e-5, 0)
    with torch.no_grad():
        plain = mf.mlp3_ln(srcs, segs, p[:3], p[3:6], act, p[6], p[7], 1e-5, 0)
    out.backward(up.cuda())
    assert torch.equal(out, plain)                       # keeping the pre-activations does not change the result
    # bf16 operands (2^-9 each) through three products and one rounding of the result: measured 3e-3
    assert _rel(out.cpu(), ref.detach()) < 8e-3
    for name, a, b in zip("edge node w1 w2 w3 b1 b2 b3 gamma beta".split(), dev, leaves):
        if b.grad is None or float(b.grad.norm()) == 0.0:
            continue
        # gradients see two more roundings per layer; ReLU also flips the sign of pre-activations near zero (one row in 100),
        # and a single row has no averaging over rows
        tol = 0.06 if rows < 64 or act == 3 else 0.02
        assert _rel(a.grad.cpu(), b.grad) < tol, name
    assert ops.device_error() == 0


@pytest.mark.gpu
def test_mlp3_ln_takes_the_same_calls_as_the_layered_path():
    """Strided tables, odd alignments and other widths keep their answers: by the one kernel or layer by layer."""
    from physicsnemo_b200.nn.module.gnn_layers.mesh_graph_mlp import MeshGraphMLP
    from physicsnemo_b200.ops import mlp_fused as mf

    torch.manual_seed(0)
    m = MeshGraphMLP(W, W, W, 2, torch.nn.SiLU()).cuda()
    wide = torch.randn(300, 2 * W + 8, device="cuda").bfloat16()
    for x, one in ((wide[:, :W].contiguous(), True), (torch.randn(300, 3 * W, device="cuda").bfloat16()[:, W:2 * W], True),
                   (wide[:, 8:8 + W], False), (wide[:0, :W].contiguous(), False)):
        layers = [m.model[0].weight, m.model[2].weight, m.model[4].weight], [m.model[i].bias for i in (0, 2, 4)]
        assert mf.supported([x], [None], *layers, [2, 2, 0], m.model[5].weight, m.model[5].bias, None) is one
        if x.shape[0]:
            with torch.autocast("cuda", dtype=torch.bfloat16), torch.no_grad():
                y = m(x)
            assert _rel(y.cpu(), m.double()(x.double()).detach().cpu()) < 1e-2
            m.float()


@pytest.mark.gpu
def test_mlp3_ln_under_activation_checkpointing():
    """Checkpointing recomputes the forward and unpacks every saved tensor once: same gradients as without."""
    from torch.utils.checkpoint import checkpoint

    from physicsnemo_b200.nn.module.gnn_layers.graph_types import Graph
    from physicsnemo_b200.nn.module.gnn_layers.mesh_edge_block import MeshEdgeBlock
    from physicsnemo_b200.nn.module.gnn_layers.mesh_node_block import MeshNodeBlock

    torch.manual_seed(0)
    edge, node = MeshEdgeBlock(W, W, W, W, 2).cuda(), MeshNodeBlock("mean", W, W, W, W, 2).cuda()
    graph = Graph(torch.randint(0, 301, (2, 1500)).cuda(), num_nodes=301)
    e, v = torch.randn(1500, W, device="cuda").bfloat16(), torch.randn(301, W, device="cuda").bfloat16()
    grads = []
    for wrap in (lambda f, *a: f(*a), lambda f, *a: checkpoint(f, *a, use_reentrant=False)):
        leaves = [e.clone().requires_grad_(), v.clone().requires_grad_()]
        params = [*edge.parameters(), *node.parameters()]
        for p in params:
            p.grad = None
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = wrap(lambda a, b: node(*edge(a, b, graph), graph), *leaves)
        torch.autograd.backward(out, [torch.ones_like(t) for t in out])
        grads.append([t.grad.clone() for t in (*leaves, *params)])
    for a, b in zip(*grads):
        # the same kernels on the same values; only the order of fp32 atomic additions differs
        assert _rel(a, b.double()) < 1e-4


@pytest.mark.gpu
def test_split_segment_sums_keep_the_fp32_sum_and_its_infinities():
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf
    from physicsnemo_b200.ops import gemm as G

    x = torch.randn(500, W, device="cuda").bfloat16()
    index = torch.arange(500, device="cuda") % 7                       # segments 7, 8 and 9 are empty
    x[0, :4] = torch.tensor([float("inf"), -float("inf"), float("nan"), 3.3e38], device="cuda").bfloat16()
    x[7, 3] = 3.3e38                                                   # finite rows whose sum is not
    seg = ops.SegmentIndex(index, 10)
    out = torch.empty(10, 2 * W, dtype=torch.bfloat16, device="cuda")
    rc = mf._lib_mlp().pnm_segment_sum_split(x.data_ptr(), seg.perm.data_ptr(), seg.offsets.data_ptr(), out.data_ptr(), 2 * W, 10, W, G._stream())
    assert rc == 0
    got = out[:, :W].double() + out[:, W:].double()
    ref = torch.zeros(10, W, device="cuda", dtype=torch.float64).index_add_(0, index, x.double())
    assert torch.isposinf(got[0, 0]) and torch.isneginf(got[0, 1]) and torch.isnan(got[0, 2]) and torch.isposinf(got[0, 3])
    got[0, :4] = ref[0, :4] = 0
    # two bf16 parts carry 16 bits of the sum
    assert float((got - ref).abs().max()) <= 2 ** -16 * float(ref.abs().max()) + 1e-5


@pytest.mark.gpu
def test_mlp3_backward_beside_other_work():
    """Many tiles per CTA while other kernels share the SMs and the memory, so that the roles of a CTA run at other speeds: every
    pass gives the sums of the first, and no wait runs out."""
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    rows = 148 * 128 * 9 + 65
    x, up = (torch.randn(rows, W, device="cuda").bfloat16() for _ in range(2))
    p = [t.cuda().requires_grad_() for t in (*(torch.randn(W, W) / W ** 0.5 for _ in range(3)), *(0.1 * torch.randn(W) for _ in range(3)),
                                             1 + 0.1 * torch.randn(W), 0.1 * torch.randn(W))]
    big = torch.randn(1 << 26, device="cuda")
    side, first = torch.cuda.Stream(), None
    for k in range(25):
        with torch.cuda.stream(side):
            for _ in range(k % 4):
                big.mul_(1.0)
        leaf = x.clone().requires_grad_()
        grads = torch.autograd.grad(mf.mlp3_ln([leaf], [None], p[:3], p[3:6], 2, p[6], p[7], 1e-5, 0), [leaf, *p], up)
        first = first or grads
        assert torch.equal(grads[0], first[0])
        # sums over rows: the same addends, another order of the fp32 additions of the CTAs
        assert all(_rel(a, b.double()) < 1e-5 for a, b in zip(grads[1:], first[1:]))
    torch.cuda.synchronize()
    assert ops.device_error() == 0


@pytest.mark.gpu
def test_mlp3_ln_without_gradients_keeps_forward_mode_and_tracing_honest():
    from torch.autograd import forward_ad

    from physicsnemo_b200.nn.module.gnn_layers.mesh_graph_mlp import MeshGraphMLP

    m = MeshGraphMLP(W, W, W, 2, torch.nn.SiLU()).cuda().requires_grad_(False)
    x, other = (torch.randn(300, W, device="cuda").bfloat16() for _ in range(2))
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), torch.no_grad():
        want = m(other)
        traced = torch.jit.trace(lambda a: m(a), (x,), check_trace=False)
        assert torch.equal(traced(other), want)
        with forward_ad.dual_level(), pytest.raises((NotImplementedError, RuntimeError)):
            m(forward_ad.make_dual(x, other))


@pytest.mark.gpu
def test_mlp3_keeps_the_moments_of_the_rows_that_the_backward_reads():
    from physicsnemo_b200.ops import mlp_fused as mf

    x = torch.randn(5000, W, device="cuda").bfloat16()
    p = [torch.randn(W, W, device="cuda") / W ** 0.5 for _ in range(3)] + [0.1 * torch.randn(W, device="cuda") for _ in range(5)]
    _, (h1, h2, x3, mean, rstd, *_) = mf._forward([x], [None], p[:3], p[3:6], 2, p[6], p[7], 1e-5, None, True)
    ref = x3.double()
    # fp32 moments of exactly these values
    assert float((mean.double() - ref.mean(1)).abs().max()) < 1e-6 * float(ref.abs().max())
    assert float((rstd.double() / torch.rsqrt(ref.var(1, unbiased=False) + 1e-5) - 1).abs().max()) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("act", [1, 2, 3])
def test_mlp3_weight_gradients_are_as_exact_as_layer_by_layer(act):
    """The operands of the weight gradients are those of the forward products, rounded once: the error against 64 bits is that of the
    layered path (16 384 entries a matrix and four draws: the ratio scatters by half a per cent; operands rounded twice give 1.08)."""
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    err = {"one": [0.0] * 3, "layered": [0.0] * 3}
    for draw in range(4):
        x, up = (torch.randn(6001, W, device="cuda").bfloat16() for _ in range(2))
        p = [torch.randn(W, W, device="cuda") / W ** 0.5 for _ in range(3)] + [0.1 * torch.randn(W, device="cuda") for _ in range(3)]
        p += [1 + 0.1 * torch.randn(W, device="cuda"), 0.1 * torch.randn(W, device="cuda")]
        q = [t.double().requires_grad_() for t in p]
        h = ACTS[act](F.linear(ACTS[act](F.linear(x.double(), q[0], q[3])), q[1], q[4]))
        ref = torch.autograd.grad(F.layer_norm(F.linear(h, q[2], q[5]), (W,), q[6], q[7]), q[:3], up.double())
        for name in err:
            w = [t.clone().requires_grad_() for t in p]
            if name == "one":
                y = mf.mlp3_ln([x], [None], w[:3], w[3:6], act, w[6], w[7], 1e-5, None)
            else:
                y = ops.layer_norm(ops.mlp_chain(x, w[:3], w[3:6], [act, act, 0]), w[6], w[7])
            for k, (g, r) in enumerate(zip(torch.autograd.grad(y, w[:3], up), ref)):
                err[name][k] += _rel(g, r)
    for one, layered in zip(err["one"], err["layered"]):
        assert one < 1.03 * layered


@pytest.mark.gpu
def test_relu_backward_drops_infinities_of_inactive_units():
    """As layer by layer: the derivative selects.  Positive matrices make every unit's gradient infinite; one unit is active."""
    from physicsnemo_b200.ops import gemm as G
    from physicsnemo_b200.ops import mlp_fused as mf

    m, dev = 200, "cuda"
    dx3 = torch.full((m, W), 3e38, device=dev).bfloat16()
    h2, h1 = torch.zeros(m, W, device=dev).bfloat16(), torch.zeros(m, W, device=dev).bfloat16()
    h2[:, 5] = h1[:, 7] = 1.0
    w = torch.ones(W, W, device=dev).bfloat16()
    g1 = torch.empty(m, W, dtype=torch.bfloat16, device=dev)
    dw, db = torch.zeros(2, W, W, device=dev), torch.zeros(2, W, device=dev)
    rc = mf._lib_mlp().pnm_mlp3_bwd(dx3.data_ptr(), h2.data_ptr(), h1.data_ptr(), h2.data_ptr(), h1.data_ptr(), w.data_ptr(), w.data_ptr(),
                                    G.ACT_RELU, g1.data_ptr(), dw[0].data_ptr(), dw[1].data_ptr(), db[0].data_ptr(), db[1].data_ptr(), m,
                                    G._stream())
    assert rc == 0
    want = torch.zeros(m, W, device=dev)
    want[:, 7] = float("inf")
    assert torch.equal(g1.float(), want)


@pytest.mark.gpu
def test_mlp3_gradients_hold_no_other_memory():
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    e, v = torch.randn(5000, W, device="cuda").bfloat16(), torch.randn(700, W, device="cuda").bfloat16()
    seg = ops.SegmentIndex(torch.randint(0, 700, (5000,), device="cuda"), 700)
    p = [torch.randn(W, k, device="cuda") / W for k in (3 * W, W, W)] + [torch.randn(W, device="cuda") for _ in range(5)]
    p = [t.requires_grad_() for t in p]
    mf.mlp3_ln([e, v, v], [None, seg, seg], p[:3], p[3:6], 2, p[6], p[7], 1e-5, 0).float().square().sum().backward()
    held = {t.grad.untyped_storage().data_ptr(): t.grad.untyped_storage().nbytes() for t in p}
    assert sum(held.values()) == sum(t.grad.numel() * 4 for t in p)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["two tables", "indexed only", "one indexed, no biases", "table twice and once"])
def test_mlp3_ln_sources_and_missing_vectors(form):
    """Sources by index and row by row in every mixture, without biases and shift, against 64 bits."""
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    rows, gen = 9001, torch.Generator().manual_seed(3)
    rn = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    tables = [rn(rows, W).bfloat16(), rn(700, W).bfloat16(), rn(311, W).bfloat16()]
    index = [None, torch.randint(0, 700, (rows,), generator=gen), torch.randint(0, 311, (rows,), generator=gen)]
    use, vectors = {"two tables": ([(0, 0), (1, 1), (2, 2)], True), "indexed only": ([(1, 1), (2, 2)], True),
                    "one indexed, no biases": ([(1, 1)], False), "table twice and once": ([(2, 2), (0, 0), (2, 2)], True)}[form]
    n = len(use)
    params = [rn(W, W * n) / (W * n) ** 0.5, rn(W, W) / W ** 0.5, rn(W, W) / W ** 0.5, 1 + 0.1 * rn(W)]
    params += [0.1 * rn(W) for _ in range(4)] if vectors else []
    up = rn(rows, W).bfloat16()
    ref_t, ref_p = [t.double().requires_grad_() for t in tables], [t.double().requires_grad_() for t in params]
    w1, w2, w3, ga, b1, b2, b3, be = [*ref_p, None, None, None, None][:8]
    x = torch.cat([ref_t[t] if index[i] is None else ref_t[t][index[i]] for t, i in use], 1)
    ref = F.layer_norm(F.linear(F.gelu(F.linear(F.gelu(F.linear(x, w1, b1)), w2, b2)), w3, b3), (W,), ga, be)
    ref.backward(up.double())
    got_t, got_p = [t.cuda().requires_grad_() for t in tables], [t.cuda().requires_grad_() for t in params]
    w1, w2, w3, ga, b1, b2, b3, be = [*got_p, None, None, None, None][:8]
    seg = [None if i is None else ops.SegmentIndex(i.cuda(), tables[k].shape[0]) for k, i in enumerate(index)]
    srcs, segs = [got_t[t] for t, _ in use], [seg[i] for _, i in use]
    assert mf.supported(srcs, segs, [w1, w2, w3], [b1, b2, b3], [1, 1, 0], ga, be, None)
    out = mf.mlp3_ln(srcs, segs, [w1, w2, w3], [b1, b2, b3], 1, ga, be, 1e-5, None)
    out.backward(up.cuda())
    # as in the test of the three usual forms
    assert _rel(out.detach().cpu(), ref.detach()) < 8e-3
    for a, b in zip((*got_t, *got_p), (*ref_t, *ref_p)):
        assert (a.grad is None) == (b.grad is None) and (b.grad is None or _rel(a.grad.cpu(), b.grad) < 0.02)
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("aggregation", ["sum", "mean"])
@pytest.mark.parametrize("checkpointed", [False, True])
def test_message_passing_step_against_64_bits(aggregation, checkpointed):
    from torch.utils.checkpoint import checkpoint

    from physicsnemo_b200.nn.module.gnn_layers.graph_types import Graph
    from physicsnemo_b200.nn.module.gnn_layers.mesh_edge_block import MeshEdgeBlock
    from physicsnemo_b200.nn.module.gnn_layers.mesh_node_block import MeshNodeBlock

    edge, node = MeshEdgeBlock(W, W, W, W, 2).cuda(), MeshNodeBlock(aggregation, W, W, W, W, 2).cuda()
    index = torch.randint(0, 301, (2, 1500)).cuda()
    e, v = torch.randn(1500, W, device="cuda").bfloat16(), torch.randn(301, W, device="cuda").bfloat16()
    ups = [torch.randn(1500, W, device="cuda").bfloat16(), torch.randn(301, W, device="cuda").bfloat16()]
    results = []
    for exact in (False, True):
        if exact:
            edge, node = edge.double(), node.double()
        for p in (*edge.parameters(), *node.parameters()):
            p.grad = None
        graph = Graph(index, num_nodes=301)
        leaves = [(t.double() if exact else t.clone()).requires_grad_() for t in (e, v)]
        step = lambda a, b: node(*edge(a, b, graph), graph)  # noqa: E731
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=not exact):
            out = checkpoint(step, *leaves, use_reentrant=False) if checkpointed and not exact else step(*leaves)
        torch.autograd.backward(out, [t.to(o.dtype) for t, o in zip(ups, out)])
        results.append([t.detach().clone() for t in out] + [t.grad.clone() for t in leaves] + [p.grad.clone() for p in (*edge.parameters(), *node.parameters())])
    for k, (a, b) in enumerate(zip(*results)):
        # outputs: four bf16 roundings; gradients: 0.8 % at this size with 128 entries in a bias
        assert _rel(a, b.double()) < (8e-3 if k < 2 else 0.02)


@pytest.mark.gpu
@pytest.mark.parametrize("act", [1, 2, 3])
@pytest.mark.parametrize("rows", [77, 3 * 148 * 128 + 5])
def test_mlp3_products_add_their_terms_in_the_order_of_the_plain_product(rows, act):
    """Bit for bit what the layered products give from the same operands: no column of an operand changes its place in a sum."""
    from physicsnemo_b200.ops import gemm as G
    from physicsnemo_b200.ops import mlp_fused as mf

    x = torch.randn(rows, W, device="cuda").bfloat16()
    w = [(torch.randn(W, W, device="cuda") / W ** 0.5).bfloat16() for _ in range(3)]
    b = [0.1 * torch.randn(W, device="cuda") for _ in range(3)]
    gamma, beta = 1 + 0.1 * torch.randn(W, device="cuda"), 0.1 * torch.randn(W, device="cuda")
    y, (h1, h2, x3, *_) = mf._forward([x], [None], w, b, act, gamma, beta, 1e-5, None, True)
    assert torch.equal(h1, G.gemm_tn(x, w[0], bias=b[0], act=act))
    assert torch.equal(h2, G.gemm_tn(h1, w[1], bias=b[1], act=act))
    assert torch.equal(x3, G.gemm_tn(h2, w[2], bias=b[2]))
    plain, _ = mf._forward([x], [None], w, b, act, gamma, beta, 1e-5, None, False)
    assert torch.equal(y, plain)


@pytest.mark.gpu
@pytest.mark.parametrize("act", [2, 3])
def test_mlp3_ln_many_tiles_per_cta(act):
    """Eight tiles and more per CTA, from three sources of which two are indexed: every accumulator, ring slot and barrier parity comes
    round again.  Against 64 bits row by row, and the same beside other kernels that make a CTA's roles run at other speeds."""
    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import mlp_fused as mf

    rows, nodes = 148 * 128 * 8 + 77, 20011
    rn = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    edge, node, up = rn(rows, W).bfloat16(), rn(nodes, W).bfloat16(), rn(rows, W).bfloat16()
    index = [torch.randint(0, nodes, (rows,), device="cuda") for _ in range(2)]
    params = [rn(W, 3 * W) / (3 * W) ** 0.5, rn(W, W) / W ** 0.5, rn(W, W) / W ** 0.5, *(0.1 * rn(W) for _ in range(3)), 1 + 0.1 * rn(W), 0.1 * rn(W)]
    segs = [None] + [ops.SegmentIndex(i, nodes) for i in index]

    leaves = [t.double().requires_grad_() for t in (edge, node, *params)]
    e, v, w1, w2, w3, b1, b2, b3, ga, be = leaves
    h = ACTS[act](F.linear(ACTS[act](F.linear(torch.cat([e, v[index[0]], v[index[1]]], 1), w1, b1)), w2, b2))
    ref = F.layer_norm(F.linear(h, w3, b3), (W,), ga, be) + e
    want = torch.autograd.grad(ref, leaves, up.double())
    ref = ref.detach()
    del h

    big, side, first = rn(1 << 26), torch.cuda.Stream(), None
    torch.cuda.synchronize()
    for k in range(9):
        with torch.cuda.stream(side):
            for _ in range(k % 3):
                big.mul_(1.0)
        dev = [t.clone().requires_grad_() for t in (edge, node, *params)]
        e, v, *p = dev
        out = mf.mlp3_ln([e, v, v], segs, p[:3], p[3:6], act, p[6], p[7], 1e-5, 0)
        with torch.no_grad():
            plain = mf.mlp3_ln([e, v, v], segs, p[:3], p[3:6], act, p[6], p[7], 1e-5, 0)
        assert torch.equal(out, plain)
        got = torch.autograd.grad(out, dev, up)
        if first is None:
            first = out.detach()
            # a row's error: 3e-3 on average as in the other tests, a few of its 128 values more; a row from another tile is off by 1
            assert float(((first.double() - ref).norm(dim=1) / ref.norm(dim=1)).max()) < 0.03
        assert torch.equal(out, first)
        for a, b in zip(got, want):                          # ReLU: pre-activations near zero, as above
            assert _rel(a, b) < (0.06 if act == 3 else 0.02)
    torch.cuda.synchronize()
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("act", [torch.nn.SiLU, torch.nn.ReLU, torch.nn.GELU])
@pytest.mark.parametrize("nsrc,post", [(1, None), (2, 1), (3, 0)])
def test_call_from_the_modules_is_the_general_call(act, nsrc, post):
    """The native walk over a Sequential gives what ``mlp3_ln`` gives, bit for bit, and declines what it does not know: a first call
    (no copies of the weights yet), weights changed in place, another stream, a subclass, another form of an activation."""
    from torch import nn

    from physicsnemo_b200 import ops
    from physicsnemo_b200.ops import gemm as G
    from physicsnemo_b200.ops import mlp_fused as mf

    torch.manual_seed(nsrc)
    mods = [nn.Linear(nsrc * W, W), act(), nn.Linear(W, W), act(), nn.Linear(W, W), nn.LayerNorm(W)]
    model = nn.Sequential(*mods).cuda()
    n, m = 300, 777
    srcs = [torch.randn(m if j == 0 else n, W, device="cuda").bfloat16() for j in range(nsrc)] if nsrc == 3 else \
        [torch.randn(m, W, device="cuda").bfloat16() for _ in range(nsrc)]
    segs = [None] + [ops.SegmentIndex(torch.randint(0, n, (m,), device="cuda"), n) for _ in range(2)] if nsrc == 3 else [None] * nsrc
    p = None if post is None else srcs[post]
    code = {nn.SiLU: G.ACT_SILU, nn.ReLU: G.ACT_RELU, nn.GELU: G.ACT_GELU}[act]
    lin = [mods[0], mods[2], mods[4]]

    def general():
        return mf.mlp3_ln(srcs, segs, [q.weight for q in lin], [q.bias for q in lin], code, mods[5].weight, mods[5].bias, mods[5].eps, post)

    with torch.no_grad():
        assert mf.module_call(model, srcs, segs, p) is None                     # no copies yet
        want = general()
        assert torch.equal(mf.module_call(model, srcs, segs, p), want)
        mods[2].weight.mul_(1.5)
        assert mf.module_call(model, srcs, segs, p) is None                     # the copy is of the values before
        want = general()
        assert torch.equal(mf.module_call(model, srcs, segs, p), want)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            assert mf.module_call(model, srcs, segs, p) is None                 # each stream has its own copies
        torch.cuda.current_stream().wait_stream(side)
        if p is not None:
            assert mf.module_call(model, srcs, segs, p.clone()) is None         # the residual is none of the tables
        assert mf.module_call(model, [t[:, :64] for t in srcs], segs, None) is None
        if act is nn.GELU:
            mods[1].approximate = "tanh"
            assert mf.module_call(model, srcs, segs, p) is None
            mods[1].approximate = "none"

        class Other(nn.Linear):
            pass

        model[4] = Other(W, W).cuda()
        assert mf.module_call(model, srcs, segs, p) is None
    with torch.enable_grad():
        assert mf.module_call(model, srcs, segs, p) is None
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("at", ["bias", "beta"])
def test_vectors_of_another_length_are_declined(at):
    """The kernel reads 128 values of every vector: a shorter one is left to the general way, from the modules and by `supported`."""
    from torch import nn

    from physicsnemo_b200.ops import gemm as G
    from physicsnemo_b200.ops import mlp_fused as mf

    model = nn.Sequential(nn.Linear(W, W), nn.SiLU(), nn.Linear(W, W), nn.SiLU(), nn.Linear(W, W), nn.LayerNorm(W)).cuda()
    lin, norm, x = [model[0], model[2], model[4]], model[5], torch.randn(40, W, device="cuda").bfloat16()

    def supported():
        return mf.supported([x], [None], [q.weight for q in lin], [q.bias for q in lin], (G.ACT_SILU, G.ACT_SILU, 0), norm.weight, norm.bias, None)

    with torch.no_grad():
        assert supported()
        mf.mlp3_ln([x], [None], [q.weight for q in lin], [q.bias for q in lin], G.ACT_SILU, norm.weight, norm.bias, norm.eps, None)
        assert mf.module_call(model, [x], [None], None) is not None
        (norm if at == "beta" else lin[1]).bias = nn.Parameter(torch.zeros(1, device="cuda"))
        assert not supported() and mf.module_call(model, [x], [None], None) is None
