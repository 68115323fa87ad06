"""What is timed: the building blocks of the framework's four benchmark models, and one model as a whole.

The networks that users of this framework train and serve are MeshGraphNet (meshes), Transolver (point clouds), AFNO
(global weather grids) and the EDM SongUNet (diffusion on images).  Nearly all of their time goes into one repeated block
each, so a case is one such block, called through its public module under bf16 autocast, forward only (serving) or
forward and backward with the gradients of the inputs and of every parameter (training).  Widths are those of the
benchmark configurations; the number of nodes, points, tokens or pixels runs from a single small sample to a full one.

Weights are drawn by the same seeded generator that makes the inputs and are written into the modules, so that ``exact``
can state every result in 64 bits with plain torch operators and without the package.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

BF16 = torch.bfloat16
DEV = "cuda"

#: widths of the benchmark configurations
MGN_WIDTH = 128
TRANSOLVER = dict(dim=256, heads=8, slices=64, ratio=4)
AFNO = dict(dim=768, blocks=8, ratio=4, threshold=0.01)
EMB = 512                    # width of the noise embedding of the 128-channel SongUNet


def listed() -> list[dict]:
    return [
        # one message-passing step on a cylinder-flow mesh of a couple of thousand nodes: the inner step of a roll-out
        dict(name="mgn_small_infer", kind="mgn_layer", nodes=1885, train=False, act="relu"),
        # a step on one ragged partition of a mesh, training
        dict(name="mgn_ragged_train", kind="mgn_layer", nodes=30011, train=True, act="silu"),
        # a step of the two-million-node benchmark mesh cut into eight parts, serving and training
        dict(name="mgn_large_infer", kind="mgn_layer", nodes=250000, train=False, act="silu"),
        dict(name="mgn_large_train", kind="mgn_layer", nodes=250000, train=True, act="silu"),
        # a whole network (encoders, 15 steps, decoder) on a mid-sized mesh: prediction
        dict(name="mgn_model_infer", kind="mgn_model", nodes=10007, train=False, act="silu"),
        # a Transolver block on a small cloud (a surface patch; latency of a prediction)
        dict(name="transolver_small_infer", kind="transolver", points=4096, train=False),
        # on a car-sized cloud whose size divides nothing, training
        dict(name="transolver_odd_train", kind="transolver", points=100003, train=True),
        # on the million points of the benchmark, training
        dict(name="transolver_large_train", kind="transolver", points=1000000, train=True),
        # an AFNO block on the 720 x 1440 grid with 8 x 8 patches, two samples, training
        dict(name="afno_train", kind="afno", batch=2, h=90, w=180, train=True),
        # the same block on a coarser grid, one sample: an ensemble member's forecast step
        dict(name="afno_small_infer", kind="afno", batch=1, h=45, w=90, train=False),
        # a residual block of the U-Net's upper levels, training
        dict(name="unet_train", kind="unet", batch=1, cin=256, cout=128, res=512, attention=False, train=True),
        # the bottleneck block with attention over 64 x 64 pixels: a denoising step of the sampler
        dict(name="unet_attention_infer", kind="unet", batch=1, cin=512, cout=512, res=64, attention=True, train=False),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["mgn_layer", "mgn_layer", "transolver", "transolver", "afno", "unet"])
    train = rng.random() < 0.6
    if kind == "mgn_layer":
        return dict(kind=kind, nodes=_log_int(rng, 500, 250000), train=train,
                    act="silu" if train else rng.choice(["silu", "relu"]))
    if kind == "transolver":
        return dict(kind=kind, points=_log_int(rng, 1000, 1000000), train=train)
    if kind == "afno":
        h = rng.choice([30, 45, 60, 90])
        return dict(kind=kind, batch=rng.choice([1, 2]), h=h, w=2 * h, train=train)
    attention = rng.random() < 0.3
    if attention:
        return dict(kind=kind, batch=rng.choice([1, 2]), cin=512, cout=512, res=8 * rng.randint(3, 7), attention=True,
                    train=train)
    cin, cout = rng.choice([(128, 128), (256, 128), (256, 256), (512, 256), (512, 512)])
    return dict(kind=kind, batch=rng.choice([1, 2]), cin=cin, cout=cout, res=rng.choice([64, 96, 120, 128, 200, 256]),
                attention=False, train=train)


# --------------------------------------------------------------------------------------------------- seeded material
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


def _linear(g, name: str, n_out: int, n_in: int, bias: bool = True) -> dict:
    """A linear layer with the spread of a trained one: unit gain, small biases."""
    p = {f"{name}.weight": _randn(g, n_out, n_in) / math.sqrt(n_in)}
    if bias:
        p[f"{name}.bias"] = 0.1 * _randn(g, n_out)
    return p


def _norm(g, name: str, n: int) -> dict:
    return {f"{name}.weight": 1 + 0.1 * _randn(g, n), f"{name}.bias": 0.1 * _randn(g, n)}


def _mlp(g, name: str, n_in: int, width: int, n_out: int, norm: bool = True) -> dict:
    """Linear, act, Linear, act, Linear[, LayerNorm] under the keys of ``MeshGraphMLP``."""
    p = {}
    for i, (a, b) in enumerate(((width, n_in), (width, width), (n_out, width))):
        p |= _linear(g, f"{name}.model.{2 * i}", a, b)
    return p | _norm(g, f"{name}.model.5", n_out) if norm else p


def _mesh_edges(g, n: int) -> torch.Tensor:
    """Directed edges of a triangulated sheet of ``n`` nodes numbered row by row, both directions, sorted by source; one
    edge in twenty (another choice for every seed) is missing, as where a mesh is coarsened or has a boundary."""
    w = max(4, int(math.isqrt(n)))
    i = torch.arange(n, device=DEV)
    col = i % w
    pairs = []
    for step, ok in ((1, col < w - 1), (w, col >= 0), (w + 1, col < w - 1)):
        a = i[ok & (i + step < n)]
        pairs.append(torch.stack((a, a + step)))
    e = torch.cat(pairs, 1)
    order = torch.argsort(torch.rand(e.shape[1], generator=g, device=DEV), stable=True)
    e = e[:, order[: e.shape[1] - e.shape[1] // 20]]
    e = torch.cat((e, e.flip(0)), 1)
    return e[:, torch.argsort(e[0] * n + e[1])].contiguous()


def _sizes(case: dict) -> int:
    """Edges of the mesh, as expected (for ``work``)."""
    n = case["nodes"]
    w = max(4, int(math.isqrt(n)))
    return int(2 * 0.95 * ((n - n / w) + (n - w) + (n - n / w - w)))


def _material(case: dict, seed: int):
    """``(parameters, inputs, gradients)``: all that the case's results follow from."""
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("mgn_layer", "mgn_model"):
        n, c = case["nodes"], MGN_WIDTH
        ei = _mesh_edges(g, n)
        e = ei.shape[1]
        if kind == "mgn_layer":
            params = _mlp(g, "edge.edge_mlp", 3 * c, c, c) | _mlp(g, "node.node_mlp", 2 * c, c, c)
            x = {"edges": _randn(g, e, c, dtype=BF16), "nodes": _randn(g, n, c, dtype=BF16)}
            grads = [_randn(g, e, c, dtype=BF16), _randn(g, n, c, dtype=BF16)] if case["train"] else []
        else:
            params = _mlp(g, "edge_encoder", 3, c, c) | _mlp(g, "node_encoder", 6, c, c) | _mlp(g, "node_decoder", c, c, 3, norm=False)
            for k in range(15):
                params |= _mlp(g, f"processor.processor_layers.{2 * k}.edge_mlp", 3 * c, c, c)
                params |= _mlp(g, f"processor.processor_layers.{2 * k + 1}.node_mlp", 2 * c, c, c)
            x = {"nodes": _randn(g, n, 6), "edges": _randn(g, e, 3)}
            grads = []
        return params, dict(x, edge_index=ei), grads
    if kind == "transolver":
        t = TRANSOLVER
        c, n, d = t["dim"], case["points"], t["dim"] // t["heads"]
        params = _norm(g, "ln_1", c) | {"Attn.temperature": 0.5 + torch.rand(1, 1, t["heads"], 1, generator=g, device=DEV)}
        params |= _linear(g, "Attn.in_project_x", c, c) | _linear(g, "Attn.in_project_fx", c, c)
        params |= _linear(g, "Attn.in_project_slice", t["slices"], d) | _linear(g, "Attn.qkv_project", 3 * d, d, bias=False)
        params |= _linear(g, "Attn.out_linear", c, c) | _norm(g, "ln_mlp1.0", c)
        params |= _linear(g, "ln_mlp1.1.layers.0", t["ratio"] * c, c) | _linear(g, "ln_mlp1.1.layers.2", c, t["ratio"] * c)
        x = {"x": _randn(g, 1, n, c, dtype=BF16)}
        # a gradient that depends on the points, as a loss's does: against pure noise the temperatures' gradients cancel out
        return params, x, [(_randn(g, 1, n, c) + x["x"].float()).to(BF16)] if case["train"] else []
    if kind == "afno":
        c, nb = AFNO["dim"], AFNO["blocks"]
        bs = c // nb
        params = _norm(g, "norm1", c) | _norm(g, "norm2", c)
        for k in ("1", "2"):
            params[f"filter.w{k}"] = _randn(g, 2, nb, bs, bs) / math.sqrt(2 * bs)
            params[f"filter.b{k}"] = 0.02 * _randn(g, 2, nb, bs)
        params |= _linear(g, "mlp.fc1", AFNO["ratio"] * c, c) | _linear(g, "mlp.fc2", c, AFNO["ratio"] * c)
        shape = (case["batch"], case["h"], case["w"], c)
        return params, {"x": _randn(g, *shape, dtype=BF16)}, [_randn(g, *shape, dtype=BF16)] if case["train"] else []
    if kind == "unet":
        ci, co, r = case["cin"], case["cout"], case["res"]

        def conv(name, n_out, n_in, k):
            return {f"{name}.weight": _randn(g, n_out, n_in, k, k) / math.sqrt(n_in * k * k), f"{name}.bias": 0.1 * _randn(g, n_out)}

        params = _norm(g, "norm0", ci) | conv("conv0", co, ci, 3) | _linear(g, "affine", co, EMB) | _norm(g, "norm1", co)
        params |= conv("conv1", co, co, 3)
        if ci != co:
            params |= conv("skip", co, ci, 1)
        if case["attention"]:
            params |= _norm(g, "attn.norm", co) | conv("attn.qkv", 3 * co, co, 1) | conv("attn.proj", co, co, 1)
        image = lambda ch: _randn(g, case["batch"], ch, r, r, dtype=BF16).contiguous(memory_format=torch.channels_last)  # noqa: E731
        x = {"x": image(ci), "emb": _randn(g, case["batch"], EMB, dtype=BF16)}
        return params, x, [image(co)] if case["train"] else []
    raise ValueError(kind)


# ------------------------------------------------------------------------------------------------- the framework's side
class _Step(torch.nn.Module):
    """One message-passing step: edge update, then node update."""

    def __init__(self, act):
        super().__init__()
        from physicsnemo_b200.nn.module.gnn_layers.mesh_edge_block import MeshEdgeBlock
        from physicsnemo_b200.nn.module.gnn_layers.mesh_node_block import MeshNodeBlock

        c = MGN_WIDTH
        self.edge = MeshEdgeBlock(c, c, c, c, 2, act)
        self.node = MeshNodeBlock("sum", c, c, c, c, 2, act)

    def forward(self, edges, nodes, graph):
        edges, nodes = self.edge(edges, nodes, graph)
        return self.node(edges, nodes, graph)


def _module(case: dict) -> torch.nn.Module:
    kind = case["kind"]
    if kind == "mgn_layer":
        return _Step({"silu": torch.nn.SiLU, "relu": torch.nn.ReLU}[case["act"]]())
    if kind == "mgn_model":
        from physicsnemo_b200.models.meshgraphnet import MeshGraphNet

        return MeshGraphNet(input_dim_nodes=6, input_dim_edges=3, output_dim=3, processor_size=15, mlp_activation_fn=case["act"],
                            hidden_dim_processor=MGN_WIDTH, aggregation="sum")
    if kind == "transolver":
        from physicsnemo_b200.models.transolver.transolver import TransolverBlock

        t = TRANSOLVER
        return TransolverBlock(t["heads"], t["dim"], 0.0, act="gelu", mlp_ratio=t["ratio"], slice_num=t["slices"], use_te=False)
    if kind == "afno":
        from physicsnemo_b200.models.afno.afno import Block

        return Block(AFNO["dim"], AFNO["blocks"], float(AFNO["ratio"]), sparsity_threshold=AFNO["threshold"])
    from physicsnemo_b200.nn.module.unet_layers import UNetBlock

    return UNetBlock(case["cin"], case["cout"], EMB, attention=case["attention"], num_heads=1, skip_scale=math.sqrt(0.5), eps=1e-6,
                     resample_proj=True, adaptive_scale=False, fused_conv_bias=True, amp_mode=True)


#: Models of earlier states.  The package recognises a parameter's bf16 copy by the parameter's identity and address; a
#: program keeps the models it has built, and so does this one.
_MODELS: list = []


def prepare(case: dict, seed: int) -> dict:
    params, x, grads = _material(case, seed)
    module = _module(case).to(DEV).train(case["train"])
    _MODELS.append(module)
    module.load_state_dict(params, strict=True)
    graph = None
    if "edge_index" in x:
        from physicsnemo_b200.nn.module.gnn_layers.graph_types import Graph

        graph = Graph(x.pop("edge_index"), num_nodes=case["nodes"])
    if case["train"]:
        for t in x.values():
            t.requires_grad_(True)
    return dict(case=case, module=module, x=x, graph=graph, grads=grads)


def _forward(state: dict):
    m, x, kind = state["module"], state["x"], state["case"]["kind"]
    if kind == "mgn_layer":
        return list(m(x["edges"], x["nodes"], state["graph"]))
    if kind == "mgn_model":
        return [m(x["nodes"], x["edges"], state["graph"])]
    if kind == "unet":
        return [m(x["x"], x["emb"])]
    return [m(x["x"])]


def run(state: dict):
    if not state["case"]["train"]:
        with torch.no_grad(), torch.autocast("cuda", dtype=BF16):
            return _forward(state)
    m, x = state["module"], state["x"]
    m.zero_grad(set_to_none=True)
    for t in x.values():
        t.grad = None
    with torch.autocast("cuda", dtype=BF16):
        out = _forward(state)
    torch.autograd.backward(out, state["grads"])
    return {"out": [t.detach() for t in out], "input_grads": {k: t.grad for k, t in x.items()},
            "param_grads": {k: p.grad for k, p in m.named_parameters()}}


# ------------------------------------------------------------------------------------------------- the work of a pass
def work(case: dict) -> dict:
    """Bytes: inputs (and the gradients that come from above) read once, results written once, weights in 32 bits.
    FLOPs: the products of the layers as they are defined, three times as many with the backward."""
    kind, train = case["kind"], case["train"]
    if kind in ("mgn_layer", "mgn_model"):
        n, c = case["nodes"], MGN_WIDTH
        e = _sizes(case)
        layer = 2 * e * 5 * c * c + 2 * n * 4 * c * c
        if kind == "mgn_model":
            flops = 15 * layer + 2 * e * (3 + 2 * c) * c + 2 * n * (6 + 2 * c) * c + 2 * n * (2 * c + 3) * c
            return dict(bytes=4.0 * (9 * n + 3 * e) + 16.0 * e + 4 * 15 * 9 * c * c, flops=float(flops))
        data, weights, flops = 2 * c * (e + n) * 2 + 16 * e, 4 * 9 * c * c, layer
        more = 2 * c * (e + n) * 2
    elif kind == "transolver":
        n, t = case["points"], TRANSOLVER
        c, s, d = t["dim"], t["slices"], t["dim"] // t["heads"]
        flops = 2 * n * c * (3 * c + s * 3 + 2 * t["ratio"] * c)     # projections, slices / sums / de-slicing, MLP
        data, weights = 2 * 2 * n * c, 4 * (3 * c * c + 2 * t["ratio"] * c * c + s * d + 3 * d * d)
        more = data
    elif kind == "afno":
        n, c = case["batch"] * case["h"] * case["w"], AFNO["dim"]
        bs = c // AFNO["blocks"]
        freq = case["batch"] * case["h"] * min(case["h"] // 2 + 1, case["w"] // 2 + 1)
        fft = 2 * 2.5 * n * c * math.log2(case["h"] * case["w"])
        flops = 2 * n * 2 * AFNO["ratio"] * c * c + 2 * 8 * freq * c * bs + fft
        data, weights = 2 * 2 * n * c, 4 * (2 * AFNO["ratio"] * c * c + 4 * c * bs)
        more = data
    else:
        n, ci, co = case["batch"] * case["res"] ** 2, case["cin"], case["cout"]
        flops = 2 * n * (9 * ci * co + 9 * co * co + (ci * co if ci != co else 0))
        weights = 4 * (9 * ci * co + 9 * co * co)
        if case["attention"]:
            flops += 2 * n * 4 * co * co + 4 * n * case["res"] ** 2 * co
            weights += 4 * 4 * co * co
        data = 2 * n * (ci + co)
        more = data
    if train:
        return dict(bytes=float(data + more + 2 * weights), flops=3.0 * flops)
    return dict(bytes=float(data + weights), flops=float(flops))


def tolerance(case: dict) -> dict:
    """About four times what the bf16 blocks show against 64 bits (the largest over all outputs)."""
    return {"rel": {"mgn_layer": 0.02, "mgn_model": 0.03, "transolver": 0.02, "afno": 0.03, "unet": 0.025}[case["kind"]]}


# ------------------------------------------------------------------------------------------------- the results in 64 bits
def _ln(x, p, name, eps=1e-5):
    return F.layer_norm(x, (x.shape[-1],), p[f"{name}.weight"], p[f"{name}.bias"], eps)


def _lin(x, p, name):
    return F.linear(x, p[f"{name}.weight"], p.get(f"{name}.bias"))


def _mlp64(x, p, name, act):
    h = act(_lin(x, p, f"{name}.model.0"))
    h = _lin(act(_lin(h, p, f"{name}.model.2")), p, f"{name}.model.4")
    return _ln(h, p, f"{name}.model.5") if f"{name}.model.5.weight" in p else h


def _step64(e, v, src, dst, p, edge, node, act):
    e = e + _mlp64(torch.cat((e, v[src], v[dst]), 1), p, edge, act)
    agg = torch.zeros_like(v).index_add(0, dst, e)
    return e, v + _mlp64(torch.cat((agg, v), 1), p, node, act)


def _transolver64(x, p):
    t = TRANSOLVER
    n, c, h = x.shape[1], t["dim"], t["heads"]
    y = _ln(x, p, "ln_1")
    heads = lambda name: _lin(y, p, name).reshape(n, h, c // h)  # noqa: E731
    w = torch.softmax(_lin(heads("Attn.in_project_x"), p, "Attn.in_project_slice")
                      / p["Attn.temperature"].clamp(0.5, 5).reshape(1, h, 1), -1)                       # [n, h, s]
    token = torch.einsum("nhs,nhd->hsd", w, heads("Attn.in_project_fx")) / (w.sum(0) + 1e-2)[..., None]
    q, k, v = _lin(token, p, "Attn.qkv_project").chunk(3, -1)
    token = torch.softmax(q @ k.transpose(1, 2) / math.sqrt(c // h), -1) @ v
    x = x + _lin(torch.einsum("nhs,hsd->nhd", w, token).reshape(1, n, c), p, "Attn.out_linear")
    return x + _lin(F.gelu(_lin(_ln(x, p, "ln_mlp1.0"), p, "ln_mlp1.1.layers.0")), p, "ln_mlp1.1.layers.2")


def _afno64(x, p, case):
    b, h, w, c = x.shape
    nb = AFNO["blocks"]
    y = _ln(x, p, "norm1")
    kept = min(h // 2 + 1, w // 2 + 1)           # the layer keeps as many modes along the rows as there are along the columns
    z = torch.fft.rfft2(y, dim=(1, 2), norm="ortho")[:, :, :kept].reshape(b, h, kept, nb, c // nb)
    mul = lambda a, k: torch.einsum("...ni,nio->...no", a, torch.complex(*p[f"filter.w{k}"])) + torch.complex(*p[f"filter.b{k}"])  # noqa: E731
    z = mul(z, 1)
    z = mul(torch.complex(F.relu(z.real), F.relu(z.imag)), 2)
    z = torch.complex(F.softshrink(z.real, AFNO["threshold"]), F.softshrink(z.imag, AFNO["threshold"]))
    z = F.pad(torch.view_as_real(z.reshape(b, h, kept, c)), (0, 0, 0, 0, 0, w // 2 + 1 - kept))
    y = torch.fft.irfft2(torch.view_as_complex(z), s=(h, w), dim=(1, 2), norm="ortho") + y + x
    return y + _lin(F.gelu(_lin(_ln(y, p, "norm2"), p, "mlp.fc1")), p, "mlp.fc2")


def _unet64(x, emb, p, case):
    gn = lambda t, name, eps=1e-6: F.group_norm(t, 32, p[f"{name}.weight"], p[f"{name}.bias"], eps)  # noqa: E731
    conv = lambda t, name: F.conv2d(t, p[f"{name}.weight"], p[f"{name}.bias"], padding=p[f"{name}.weight"].shape[-1] // 2)  # noqa: E731
    h = conv(F.silu(gn(x, "norm0")), "conv0")
    h = conv(F.silu(gn(h + _lin(emb, p, "affine")[:, :, None, None], "norm1")), "conv1")
    h = (h + (conv(x, "skip") if "skip.weight" in p else x)) * math.sqrt(0.5)
    if case["attention"]:
        b, c = h.shape[:2]
        # three interleaved parts per channel: q, k, v of channel j are rows 3 j, 3 j + 1, 3 j + 2 of the projection
        q, k, v = conv(gn(h, "attn.norm"), "attn.qkv").reshape(b, c, 3, -1).unbind(2)
        a = torch.softmax(q.transpose(1, 2) @ k / math.sqrt(c), -1)
        h = (conv((v @ a.transpose(1, 2)).reshape(h.shape), "attn.proj") + h) * math.sqrt(0.5)
    return h


def exact(case: dict, seed: int):
    params, x, grads = _material(case, seed)
    ei = x.pop("edge_index", None)
    train, kind = case["train"], case["kind"]
    p = {k: v.double().requires_grad_(train) for k, v in params.items()}
    x = {k: v.double().requires_grad_(train) for k, v in x.items()}
    act = {"silu": F.silu, "relu": F.relu}.get(case.get("act"))
    with torch.set_grad_enabled(train):
        if kind == "mgn_layer":
            out = list(_step64(x["edges"], x["nodes"], ei[0], ei[1], p, "edge.edge_mlp", "node.node_mlp", act))
        elif kind == "mgn_model":
            e, v = _mlp64(x["edges"], p, "edge_encoder", act), _mlp64(x["nodes"], p, "node_encoder", act)
            for k in range(15):
                layer = "processor.processor_layers.%d"
                e, v = _step64(e, v, ei[0], ei[1], p, layer % (2 * k) + ".edge_mlp", layer % (2 * k + 1) + ".node_mlp", act)
            out = [_mlp64(v, p, "node_decoder", act)]
        elif kind == "transolver":
            out = [_transolver64(x["x"], p)]
        elif kind == "afno":
            out = [_afno64(x["x"], p, case)]
        else:
            out = [_unet64(x["x"], x["emb"], p, case)]
    if not train:
        return out
    torch.autograd.backward(out, [g.double() for g in grads])
    return {"out": [t.detach() for t in out], "input_grads": {k: t.grad for k, t in x.items()},
            "param_grads": {k: t.grad for k, t in p.items()}}
