"""Launches whose CTAs meet in memory (csrc/workspace.cpp), on several streams, threads and graphs at the same time: each gives the bits that it gives alone."""
import gc
import threading

import pytest
import torch

from neuronx_distributed_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
ROUNDS = 60


def _calls(seed):
    """Stream-K GEMVs (bf16 and fp8 weights), GEMMs with a split K, split decode attention, argmax: (call, result alone) pairs."""
    g = torch.Generator(DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, dtype=BF, generator=g)
    x, w = rnd(2, 4096), rnd(5000, 4096) * 0.02
    x8, w8 = rnd(3, 8192), (rnd(2056, 8192) * 0.02).to(torch.float8_e4m3fn)
    s8 = torch.rand(2056, device=DEV, generator=g)
    q, cache, lines, pos = rnd(2, 1, 8, 128), rnd(3, 2, 4096, 128), torch.tensor([0, 1], device=DEV, dtype=torch.int32), torch.tensor([[4000], [2500]], device=DEV, dtype=torch.int32)
    xk, wk, xs, ws = rnd(200, 8192), rnd(1024, 8192) * 0.02, rnd(130, 4096), rnd(512, 4096) * 0.02
    logits = torch.randn(4, 50000, device=DEV, generator=g)
    calls = [lambda: ops.linear(x, w), lambda: ops.linear(x, w, act="silu_mul"), lambda: ops.linear(x8, w8, scale=s8), lambda: ops.linear(xk, wk), lambda: ops.linear(xs, ws, act="silu_mul"),
             lambda: ops.attention_decode(q, cache, cache, lines, pos, 0.09), lambda: ops.argmax(logits)]
    return [(f, f()) for f in calls]


def _same(results, pairs):
    return all(torch.equal(r, want) for row in results for r, (_, want) in zip(row, pairs))


def test_streams():
    work = [(torch.cuda.Stream(), _calls(s)) for s in range(3)]
    torch.cuda.synchronize()
    got = [[] for _ in work]
    for _ in range(ROUNDS):
        for k, (stream, pairs) in enumerate(work):
            with torch.cuda.stream(stream):
                got[k].append([f() for f, _ in pairs])
    torch.cuda.synchronize()
    assert all(_same(r, pairs) for r, (_, pairs) in zip(got, work))


def test_more_streams_than_are_kept():
    pairs = _calls(0)
    streams = [torch.cuda.Stream() for _ in range(20)]
    torch.cuda.synchronize()
    got = []
    for _ in range(3):
        for stream in streams:
            with torch.cuda.stream(stream):
                got.append([f() for f, _ in pairs])
    torch.cuda.synchronize()
    assert _same(got, pairs)


def test_threads():
    work = [(torch.cuda.Stream(), _calls(s), []) for s in range(4)] + [(torch.cuda.current_stream(), _calls(s), []) for s in (4, 5)]     # two on one stream
    torch.cuda.synchronize()

    def run(stream, pairs, got):
        with torch.cuda.stream(stream):
            for _ in range(ROUNDS):
                got.append([f() for f, _ in pairs])

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(len(got) == ROUNDS and _same(got, pairs) for _, pairs, got in work)


def test_graphs_beside_each_other_and_beside_eager_calls():
    work = [_calls(s) for s in range(3)]
    torch.cuda.synchronize()
    graphs = []
    for pairs in work[:2]:                               # both captured on the same side stream
        graph, out = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph):
            for f, _ in pairs * 3:
                out.append(f())
        graphs.append((graph, out, torch.cuda.Stream()))
    eager, got, seen = torch.cuda.Stream(), [], [[], []]
    torch.cuda.synchronize()
    for _ in range(ROUNDS):
        for k, (graph, out, stream) in enumerate(graphs):
            with torch.cuda.stream(stream):
                graph.replay()
                seen[k].append([o.clone() for o in out])
        with torch.cuda.stream(eager):
            got.append([f() for f, _ in work[2]])
    torch.cuda.synchronize()
    assert _same(got, work[2])
    for rows, pairs in zip(seen, work):
        assert _same(rows, pairs * 3)


def test_a_capture_with_two_branches():
    a, b = _calls(0), _calls(1)
    side = torch.cuda.Stream()
    graph, out_a, out_b = torch.cuda.CUDAGraph(), [], []
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        for (f, _), (g, _) in zip(a * 4, b * 4):
            out_a.append(f())
            with torch.cuda.stream(side):
                out_b.append(g())
        main.wait_stream(side)
    for _ in range(10):
        graph.replay()
        torch.cuda.synchronize()
        assert _same([out_a], a * 4) and _same([out_b], b * 4)


def _capture(calls, **kw):
    graph, out = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph, **kw):
        for f, _ in calls:
            out.append(f())
    return graph, out


def test_rows_of_graphs_are_given_back():
    """260 graphs at once: 256 take a row of cleared tickets, the others clear theirs; the rows are free again when the graphs are gone."""
    ext, pairs = ops._C(), _calls(0)
    pairs = [pairs[0], pairs[-1]]
    gc.collect()
    torch.cuda.synchronize()
    before = ext.workspace_rows_in_use(0)
    for _ in range(2):
        graphs = [_capture(pairs) for _ in range(260)]
        assert ext.workspace_rows_in_use(0) == 256
        for _ in range(2):
            for graph, out in graphs:
                graph.replay()
            torch.cuda.synchronize()
            assert all(_same([out], pairs) for _, out in graphs)
        del graph, out, graphs
        gc.collect()
        torch.cuda.synchronize()
        assert ext.workspace_rows_in_use(0) == before
        torch.cuda.empty_cache()
        assert ext.workspace_rows_in_use(0) == before


def test_graphs_of_one_pool_share_a_row():
    """They share their other memory too, and are replayed one after the other; the row stays until the last of them is gone."""
    ext, pairs = ops._C(), _calls(0)
    gc.collect()
    before = ext.workspace_rows_in_use(0)
    stream, pool = torch.cuda.Stream(), torch.cuda.graph_pool_handle()
    graphs = [_capture(pairs, pool=pool, stream=stream)[0] for _ in range(3)]
    assert ext.workspace_rows_in_use(0) == before + 1
    del graphs[:2]
    gc.collect()
    assert ext.workspace_rows_in_use(0) == before + 1
    more, out = _capture(pairs, pool=pool, stream=stream)
    graphs[0].replay()
    more.replay()
    torch.cuda.synchronize()
    assert _same([out], pairs) and ext.workspace_rows_in_use(0) == before + 1
    del graphs, more, out
    gc.collect()
    assert ext.workspace_rows_in_use(0) == before
