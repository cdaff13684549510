"""The native form of the tensor wrappers (``binding/calls.cpp``) against their Python form: the same results bit for
bit over the options that both take, and the same errors."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from compactattention_b200 import ops as _ops
    assert _ops._calls is not None, "the native wrappers are not built (python -m compactattention_b200.build)"
    return _ops


def _both(ops, monkeypatch, fn, *names):
    """``fn()`` through Python and then through the native form, which must have served every call, of just these names."""
    with monkeypatch.context() as m:
        m.setattr(ops, "_calls", None)
        python = fn()
    fn()  # what the wrappers keep per stream exists from here on
    seen, real = [], ops._calls

    class Watch:
        def __getattr__(self, name):
            def call(*args):
                out = getattr(real, name)(*args)
                seen.append((name, out is not None))
                return out
            return call

    with monkeypatch.context() as m:
        m.setattr(ops, "_calls", Watch())
        native = fn()
    assert [name for name, _ in seen] == list(names) and all(served for _, served in seen), seen
    return python, native


def _randn(*shape, dtype=torch.bfloat16, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda", dtype=torch.float32).to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Q", [1, 130])
def test_attention(ops, monkeypatch, dtype, Q):
    B, K, Hq, Hkv, bs = 2, 64 * 9 + Q, 8, 2, 64
    q, k, v = _randn(B, Q, Hq, 128, dtype=dtype), _randn(B, K, Hkv, 128, dtype=dtype, seed=1), _randn(B, K, Hkv, 128, dtype=dtype, seed=2)
    kv = ops.KvCacheView.from_seq_first(k, v)
    idx = torch.arange(9, dtype=torch.int32, device="cuda").repeat(B, Hkv, 1).contiguous()
    counts = torch.tensor([[9, 4], [1, 0]], dtype=torch.int32, device="cuda")
    out = torch.empty((B, Q, Hq, 136), dtype=dtype, device="cuda")[..., :128]
    for kw in ({}, {"softmax_scale": 0.05}, {"out": out}):
        a, b = _both(ops, monkeypatch, lambda: ops.attn_compact(q, kv, K, Hkv, idx, counts, block_size=bs, **kw).clone(), "attn_compact")
        assert torch.equal(a, b)
        a, b = _both(ops, monkeypatch, lambda: ops.attn_compact(q, kv, K, Hkv, None, None, block_size=bs, **kw).clone(), "attn_compact")
        assert torch.equal(a, b)
    assert ops.attn_compact(q, kv, K, Hkv, None, None, out=out) is out
    with pytest.raises(ValueError, match="share dtype"):
        ops.attn_compact(q.float(), kv, K, Hkv, None, None)
    with pytest.raises(ValueError, match="one row per"):
        ops.attn_compact(q, kv, K, Hkv, idx[:1].contiguous(), counts)
    with pytest.raises(RuntimeError, match="kv_len"):
        ops.attn_compact(q, kv, Q - 1, Hkv, None, None)


@pytest.mark.parametrize("tables", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mean", [True, False])
def test_append(ops, monkeypatch, tables, mean):
    from compactattention_b200.paged_cache import PagedKVCache
    B, Q, Hq, Hkv, pos = 2, 200, 7, 3, 128
    q, k, v = _randn(B, Q, Hq, 128), _randn(B, Q, Hkv, 128, seed=1), _randn(B, Q, Hkv, 128, seed=2)
    cos, sin = _randn(1, Q, 128, dtype=tables, seed=3), _randn(1, Q, 128, dtype=tables, seed=4)

    def run():
        cache = PagedKVCache(B, 512, Hkv, 128, torch.device("cuda"))
        mean_k = torch.zeros((B, 8, Hkv, 128), dtype=torch.bfloat16, device="cuda") if mean else None
        rot, n = cache.append_rope(q, k, v, cos, sin, position=pos, mean_k=mean_k)
        assert n == pos + Q
        return [rot, cache.k_pages, cache.v_pages] + ([mean_k] if mean else [])

    a, b = _both(ops, monkeypatch, run, "rope_append")
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    cache = PagedKVCache(B, 512, Hkv, 128, torch.device("cuda"))
    with pytest.raises(ValueError, match="do not fit in mean_k"):
        ops.rope_append(q, k, v, cos, sin, cache.view(), 128, mean_k=torch.zeros((B, 2, Hkv, 128), dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(ValueError, match="share their strides"):
        ops.rope_append(q, k, v, cos, sin.repeat(1, 1, 2)[..., :128], cache.view(), 0)


@pytest.mark.parametrize("rule,kw", [
    ("threshold", dict(threshold=0.2)),
    ("threshold", dict(threshold=0.001, softmax=True, keep_recent=3)),
    ("topk", dict(topk_ratio=(1, 5), sink=1, local=2)),
    ("topk", dict(topk_k=3)),
    ("alpha_rowmax", dict(alpha=0.5, sink=2, local=4, min_budget=5, rows_voting=2)),
    ("cummass", dict(threshold=0.6, softmax=True)),
])
@pytest.mark.parametrize("masked", [False, True])
def test_selection(ops, monkeypatch, rule, kw, masked):
    B, H, Hkv, Qb, Kb = 2, 6, 3, 4, 70
    score = _randn(B, Qb, Kb, H, dtype=torch.float32).permute(0, 3, 1, 2)  # strided, as the training-free score is
    valid = None
    if masked:
        valid = torch.ones((Qb, Kb), dtype=torch.bool, device="cuda").tril(Kb - Qb).view(1, 1, Qb, Kb)
        valid[..., 5] = False

    def run():
        t = ops.select_union_table(score, Kb - Qb, rule, num_kv_heads=Hkv, valid=valid, **kw)
        return [t.block_idx, t.counts, t.cache_seqlens, t.pages_per_row]

    a, b = _both(ops, monkeypatch, run, "select_union_table")
    assert all(torch.equal(x, y) and x.shape == y.shape for x, y in zip(a, b))
    with pytest.raises(ValueError, match="own key blocks"):
        ops.select_union_table(score, Kb - Qb - 1, rule, num_kv_heads=Hkv, **kw)
    with pytest.raises(ValueError, match="not a multiple"):
        ops.select_union_table(score, Kb - Qb, rule, num_kv_heads=4, **kw)


@pytest.mark.parametrize("rope", [True, False])
def test_gate(ops, monkeypatch, rope):
    from compactattention_b200.chunk_driver import GateSelectorState, SelectionRule
    from compactattention_b200.prefill_sparse.attn_gate import ATTNGATE_CLASSES
    Hq, Hkv, L, past = 8, 2, 300, 40
    gate = ATTNGATE_CLASSES["Qavg_Kmaxminavg"](64, 128, 128, Hkv, Hq, force_double=True).cuda().to(torch.bfloat16)
    with torch.no_grad():
        gate.mask_linear_q.weight.copy_(_randn(*gate.mask_linear_q.weight.shape, seed=5) * 0.05)
        gate.mask_linear_k.weight.copy_(_randn(*gate.mask_linear_k.weight.shape, seed=6) * 0.05)
    q, k = _randn(1, L, Hq, 128), _randn(1, L, Hkv, 128, seed=1)
    nb = -(-L // 64)
    tables = (_randn(1, nb, 128, dtype=torch.float32, seed=2), _randn(1, nb, 128, dtype=torch.float32, seed=3)) if rope else None
    rule = SelectionRule(rule="topk", softmax=False, topk_ratio=(1, 4), sink=1, local=2)
    past_blocks = _randn(1, past, Hkv, 128, seed=7)

    def run():
        st = GateSelectorState(gate, 1, torch.device("cuda"))
        st.cache.reserve(past + nb)
        st.cache.blocks_view()[:, :past].copy_(past_blocks)
        st.cache.length = past
        st.append(q, k, tables, tables)
        t = st.score_select(rule, Hkv, 64)
        return [st.q_blocks, st.cache.blocks().clone(), st.logits, t.block_idx, t.counts]

    a, b = _both(ops, monkeypatch, run, "gate_prepare", "select_union_table")
    assert all(torch.equal(x, y) for x, y in zip(a, b))


# ---- the wrappers around entry points that only note that they were called ----

FAKE = r"""
#include <unistd.h>
static int calls, code, sleep_us;
void set(int c, int us) { calls = 0, code = c, sleep_us = us; }
int count(void) { return calls; }
static int enter(void) { ++calls; usleep(sleep_us); return code; }
int one(const void* p, void* stream) { return enter(); }
int select_(const void* p, const void* u, void* s, unsigned long n, void* stream) { return enter(); }
int gate(const void* g, const void* p, const void* u, void* s, unsigned long n, int w, void* stream) { return enter(); }
int bytes(int B, int H, int Hkv, int Qb, int Kb, unsigned long* n) { *n = 16; return 0; }
const char* error(void) { return "as told"; }
"""


@pytest.fixture
def fake(ops, tmp_path):
    """The native wrappers bound to FAKE instead of the library, and one plain call through each of them."""
    import ctypes
    import subprocess
    (tmp_path / "fake.c").write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "fake.so"), str(tmp_path / "fake.c")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "fake.so"))
    native = ops._native()
    q, kv = _randn(1, 2, 4, 128), ops.KvCacheView.from_seq_first(_randn(1, 64, 2, 128), _randn(1, 64, 2, 128))
    ws = torch.empty(1024, dtype=torch.uint8, device="cuda")
    score, blocks, weight = torch.zeros((1, 4, 1, 3), device="cuda"), _randn(1, 3, 2, 128), _randn(2, 128, 128)
    qblk = torch.zeros((1, 1, 4, 128), device="cuda")
    layout = (kv.k, kv.v, kv.page_stride, kv.token_stride, kv.head_stride, kv.page_size, kv.num_pages, kv.pages_per_seq, 0, None)
    pick = (0, ws[:64].view(torch.int32), score, 2, ops.RULES["topk"], 2, 64, 256, 0, None, 0, 0.0, 0.0, 1, 0, 1, 0, 0, 0, 0, None, None, None,
            None, None)
    cs = _randn(1, 2, 128)
    calls = {
        "ca_attn_compact": lambda: native.attn_compact(0, ws, q, *layout, 64, 2, None, None, 64, None, None, None, None),
        "ca_rope_append": lambda: native.rope_append(0, q, q[:, :, :2], q[:, :, :2], cs, cs, *layout, 0, None, 64, None, None),
        "ca_gate_prepare": lambda: native.gate_prepare(0, 64, q, 4, None, None, None, qblk, 0, q[:, :, :2], 4, weight, None, None,
                                                       blocks, 0),
        "ca_select_union_table": lambda: native.select_union_table(*pick),
        "ca_gate_score_select": lambda: native.select_union_table(*pick, qblk, blocks, 1.0, 0.0, 1),
    }
    address = [ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in ("one", "one", "one", "select_", "gate", "bytes", "error")]
    assert native.bind(*address)
    yield lib, calls
    ops._native_lib = None  # the next call binds the library again


def test_a_library_error_is_raised_and_the_call_not_made_again(fake):
    lib, calls = fake
    for name, call in calls.items():
        lib.set(0, 0)
        assert call() is not None and lib.count() == 1, name
        lib.set(-3, 0)
        with pytest.raises(RuntimeError, match=rf"{name} failed \(code -3\): as told"):
            call()
        assert lib.count() == 1, name


def test_other_threads_run_while_a_call_waits(fake):
    """A launch may wait for the GPU for long; the wrappers let go of the interpreter meanwhile."""
    import threading
    lib, calls = fake
    for name, call in calls.items():
        lib.set(0, 300000)
        go, ticks = threading.Event(), []

        def tick():
            go.wait()
            for _ in range(5):  # at the earliest once the call has begun: this thread holds the GIL until then
                ticks.append(time.monotonic())
                time.sleep(0.01)

        t = threading.Thread(target=tick)
        t.start()
        go.set()
        call()
        end = time.monotonic()
        t.join()
        assert sum(x < end - 0.05 for x in ticks) == 5, name


def test_threads_on_one_stream_keep_their_pieces_apart(ops):
    """Calls whose units are cut (two launches, one workspace per stream) from several threads on one stream."""
    import threading
    cases = []
    for i, (Q, K) in enumerate(((256, 16384), (1, 60000), (300, 12000), (2, 40000))):
        q, k, v = _randn(1, Q, 4, 128, seed=i), _randn(1, K, 1, 128, seed=i + 10), _randn(1, K, 1, 128, seed=i + 20)
        kv = ops.KvCacheView.from_seq_first(k, v)
        cases.append((q, kv, K, ops.attn_compact(q, kv, K, 1, None, None).clone()))
    torch.cuda.synchronize()
    bad = []

    def work(q, kv, K, want):
        outs = [ops.attn_compact(q, kv, K, 1, None, None) for _ in range(100)]
        torch.cuda.synchronize()
        bad.append(sum(not torch.equal(o, want) for o in outs))

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == [0] * len(cases)
