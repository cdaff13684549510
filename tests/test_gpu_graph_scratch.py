"""Scratch under CUDA graphs and call recordings: a captured or recorded step shares no tickets, row bits or partials with
eager calls that run (and outgrow the buffers kept per stream) later, nor with other graphs, whatever the replay order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BS, HQ, HKV = 64, 8, 2


@pytest.fixture(scope="module")
def ops():
    from compactattention_b200 import ops as _ops
    return _ops


def _randn(*shape, seed, dtype=torch.bfloat16):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda", dtype=torch.float32).to(dtype)


def _step(kind, Q, K, seed):
    """One call of an operator (or of the wrappers that the gate layers use) -> its attention output."""
    from compactattention_b200 import ops as o
    from compactattention_b200.modules.attention_forward_chunked_dense import chunked_prefill_column_dense_attention_forward
    from compactattention_b200.modules.flashprefill_prefill import flashprefill_compactattn_prefill_full_kv
    q, k, v = (_randn(1, n, h, 128, seed=seed + i) for i, (n, h) in enumerate(((Q, HQ), (K, HKV), (K, HKV))))
    qb, kb = -(-Q // BS), -(-K // BS)
    if kind == "keep":
        score = torch.rand((1, HQ, qb, kb), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
        return lambda: chunked_prefill_column_dense_attention_forward(
            q, k, v, None, Q, attn_gate_score=score, threshold=0.97, block_size=BS, num_key_value_groups=HQ // HKV)[0]
    if kind == "flash":
        return lambda: flashprefill_compactattn_prefill_full_kv(
            q, k, v, None, softmax_scale=128 ** -0.5, num_key_value_groups=HQ // HKV, block_size=BS, attention_sink=1, window_size=2,
            alpha=0.9, last_n_block=0, min_budget=4, pack_impl="torch", indexed_impl="b200_native", cache_fill_backend="auto")[0]
    qblk, kblk = _randn(1, qb, HQ, 128, seed=seed + 3, dtype=torch.float32), _randn(1, kb, HKV, 128, seed=seed + 4)
    kv = o.KvCacheView.from_seq_first(k, v)

    def gate():
        t = o.gate_score_select(qblk, kblk, kb - qb, "topk", num_kv_heads=HKV, topk_ratio=(1, 8), sink=1, local=2)
        return o.attn_compact(q, kv, K, HKV, t.block_idx, t.counts)
    return gate


def _capture(fn, stream=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
    return graph, out


@pytest.mark.parametrize("kind", ["keep", "flash", "gate"])
def test_a_longer_call_after_the_capture(ops, kind):
    fn, longer = _step(kind, 512, 8192, 1), _step(kind, 512, 32768, 2)
    want = fn().clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    side.synchronize()
    graph, out = _capture(fn, side)
    with torch.cuda.stream(side):
        longer()  # outgrows what is kept for this stream
        words = ops._union_scratch_words(1, HQ, HKV, 8, 128)
        guards = [torch.full((words,), 0x5A5A5A5A, dtype=torch.int32, device="cuda") for _ in range(32)]
        for _ in range(3):
            out.zero_()
            graph.replay()
            side.synchronize()
            assert torch.equal(out, want)
    assert all(bool((t == 0x5A5A5A5A).all()) for t in guards)


@pytest.mark.parametrize("kind", ["keep", "flash", "gate"])
def test_the_second_capture_replayed_first(ops, kind):
    fns = [_step(kind, 512, 8192, s) for s in (3, 4)]
    wants = [fn().clone() for fn in fns]
    graphs = [_capture(fn) for fn in fns]  # torch's own capture stream, on which nothing ever ran
    for i in (1, 0, 1):
        graph, out = graphs[i]
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, wants[i])


@pytest.mark.parametrize("kind", ["keep", "flash", "gate"])
def test_graphs_of_one_stream_replayed_on_two(ops, kind):
    fns = [_step(kind, 512, 16384, s) for s in (5, 6)]
    wants = [fn().clone() for fn in fns]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for fn in fns:
            fn()
    torch.cuda.synchronize()
    graphs = [_capture(fn, side) for fn in fns]
    streams = [torch.cuda.Stream() for _ in graphs]
    same = [torch.zeros((), dtype=torch.int64, device="cuda") for _ in graphs]
    for (_, out) in graphs:
        out.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for (graph, out), st, want, n in zip(graphs, streams, wants, same):
            with torch.cuda.stream(st):
                graph.replay()
                n += (out == want).all()
    torch.cuda.synchronize()
    assert [int(n) for n in same] == [20, 20]


def test_recorded_calls_keep_their_scratch(ops):
    from compactattention_b200 import _lib
    score, longer = (torch.rand((1, HQ, 8, kb), generator=torch.Generator(device="cuda").manual_seed(kb), device="cuda") for kb in (128, 512))

    def run(s):
        return ops.select_union_table(s, s.shape[3] - 8, "topk", num_kv_heads=HKV, topk_ratio=(1, 8))

    want = run(score)
    with _lib.record() as calls:
        got = run(score)
    run(longer)
    words = ops._union_scratch_words(1, HQ, HKV, 8, 128)
    guards = [torch.full((words,), 0x5A5A5A5A, dtype=torch.int32, device="cuda") for _ in range(32)]
    for t in (got.block_idx, got.counts):
        t.zero_()
    calls.run()
    torch.cuda.synchronize()
    assert torch.equal(got.block_idx, want.block_idx) and torch.equal(got.counts, want.counts)
    assert all(bool((t == 0x5A5A5A5A).all()) for t in guards)
