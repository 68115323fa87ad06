"""The cached bf16 copy of a parameter belongs to that parameter alone."""
import gc

import torch

from physicsnemo_b200.ops import gemm as G


def test_a_new_parameter_never_gets_the_copy_of_one_that_is_gone(monkeypatch):
    a = torch.nn.Parameter(torch.full((8, 8), 1.0))
    assert G._bf16_weight(a) is G._bf16_weight(a)
    b = torch.nn.Parameter(torch.full((8, 8), 2.0))
    # as if `a` had been freed and `b` had been given its id, address and version
    (ver, val, ref), = [G._wcache[k] for k in G._wcache if k == (id(a), False)]
    monkeypatch.setitem(G._wcache, (id(b), False), ((b._version, b.data_ptr(), tuple(b.shape), b.stride()), val, ref))
    assert float(G._bf16_weight(b).float().mean()) == 2.0
    with torch.no_grad():
        b.mul_(2)                                    # a changed parameter is converted again
    assert float(G._bf16_weight(b, transpose=True).float().mean()) == 4.0


def test_views_of_one_parameter_share_its_life():
    a = torch.nn.Parameter(torch.arange(32.0).reshape(4, 2, 4))
    first = G._bf16_weight(a.reshape(4, 8))
    assert G._bf16_weight(a.reshape(4, 8)) is first and first.shape == (4, 8)
    assert G._bf16_weight(a.reshape(8, 4)).shape == (8, 4)


def test_views_used_in_turn_keep_their_copies():
    p = torch.nn.Parameter(torch.randn(3 * 8, 8))
    views = [*p.chunk(3), p[:8].t(), p]
    first = [G._bf16_weight(v) for v in views]
    assert all(G._bf16_weight(v) is f for v, f in zip(views, first))
    assert all(torch.equal(f, v.detach().bfloat16()) for v, f in zip(views, first))
    with torch.no_grad():
        p.mul_(2)
    assert all(torch.equal(G._bf16_weight(v), 2 * f) for v, f in zip(views, first))


def test_copies_go_with_their_parameter():
    gc.collect()
    before = set(G._wcache)
    p = torch.nn.Parameter(torch.randn(8, 8))
    G._bf16_weight(p), G._bf16_weight(p, transpose=True), G._bf16_weight(p[:4])
    assert len(set(G._wcache) - before) == 3
    del p
    gc.collect()
    assert set(G._wcache) <= before


def test_edge_orders_follow_the_edges():
    """The sorted orders that a graph keeps are those of its edges now: after a change in place and for an index at an old address."""
    from physicsnemo_b200.nn.module.gnn_layers.graph_types import Graph, segments

    graph = Graph(torch.tensor([[0, 1, 2], [2, 2, 0]], dtype=torch.int32), num_nodes=3)
    first = segments(graph, "dst", 3)
    assert segments(graph, "dst", 3) is first and first.counts.tolist() == [1, 0, 2]
    graph.edge_index[1] = torch.tensor([1, 1, 1])
    assert segments(graph, "dst", 3).counts.tolist() == [0, 3, 0]
    for k in range(40):                              # replaced again and again: nothing may be recognised by its address
        graph.edge_index = torch.full((2, 3), k % 3, dtype=torch.int32)
        assert segments(graph, "dst", 3).counts.tolist() == [3 * (k % 3 == n) for n in range(3)]
    assert len(graph._pnm_cache) <= 16
