"""The native host side of the per-layer calls against the Python code behind it: what it serves gives the same
bits, and what it does not serve takes the general path.  A tensor subclass is never served."""
import sys
from types import SimpleNamespace

import pytest
import torch

import workloads

pytestmark = pytest.mark.gpu


class Wrapped(torch.Tensor):
    pass


def _rows(seed, heads, tokens, dtype, form):
    """[1, heads, tokens, 128]: contiguous, token-major, a slice of a longer buffer, rows that are not 16-byte aligned."""
    x = workloads.make_kv_torch(seed, heads, max(tokens, 1), "cuda", 128)[0].to(dtype)[:, :, :tokens]
    if form == "token-major":
        return x.transpose(1, 2).contiguous().transpose(1, 2)
    if form == "slice":
        buffer = torch.zeros((1, heads, tokens + 9, 128), dtype=dtype, device="cuda")
        buffer[:, :, 5:5 + tokens] = x
        return buffer[:, :, 5:5 + tokens]
    if form == "unaligned":
        buffer = torch.zeros(heads * tokens * 128 + 1, dtype=dtype, device="cuda")
        buffer[1:] = x.reshape(-1)
        return buffer[1:].view(1, heads, tokens, 128)
    return x


@pytest.fixture
def served(monkeypatch):
    """Per native call, in order: True when it served the call, False when it left it to the Python code."""
    from inquant import _native as N
    host, calls = N.host(), {"append_token": [], "decode": [], "paged_decode": []}

    def counted(name):
        def call(*args):
            result = getattr(host, name)(*args)
            calls[name].append(result is not None)
            return result
        return call
    module = SimpleNamespace(same_objects=host.same_objects, **{name: counted(name) for name in calls})
    monkeypatch.setattr(N, "host", lambda: module)
    return calls


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["contiguous", "token-major", "slice", "unaligned"])
@pytest.mark.parametrize("value_bits,group,block", [(2, 64, 64), (None, 64, 64), (4, 32, 128), (2, 64, 48)])
def test_decode_and_append_are_those_of_the_general_path(dtype, form, value_bits, group, block):
    from inquant import _native as N
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.triton_attention import PackedDecodeState
    heads, q_heads = 2, 14
    config = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=block, residual_length=40, sink_tokens=4, value_bits=value_bits,
                         value_group_size=group, validate_positions=False)
    caches = [InQuantCache(config) for _ in range(2)]
    prompt = [_rows(s, heads, 3 + 2 * block, dtype, "contiguous") for s in (1, 2)]
    states = [None, None]
    for step in range(block // 2 + 60):
        new = [_rows(10 * step + s, heads, 1, dtype, form) for s in (3, 4)]
        query = _rows(10 * step + 5, q_heads, 1, dtype, form)
        results = []
        for i, cache in enumerate(caches):
            if not step:
                cache.update(prompt[0][:, :, :3], prompt[1][:, :, :3], 0)     # the sink is still filling
                cache.append_for_attention(*(x[:, :, 3:4] if not i else x[:, :, 3:4].as_subclass(Wrapped) for x in prompt), 0)
                cache.update(prompt[0][:, :, 4:], prompt[1][:, :, 4:], 0)
            as_given = (lambda x: x) if not i else (lambda x: x.as_subclass(Wrapped))
            view = cache.append_for_attention(*(as_given(x) for x in new), 0)
            if states[i] is None:
                states[i] = PackedDecodeState(view.key_blocks, view.value_blocks)
            elif len(states[i].key_blocks) != len(view.key_blocks):
                states[i].extend(view.key_blocks, view.value_blocks)
            dense = (view.sink_key, view.sink_value, view.residual_key, view.residual_value)
            out = states[i].decode(as_given(query), sink_key=dense[0], sink_value=dense[1], residual_key=dense[2], residual_value=dense[3])
            results.append((*(t.as_subclass(torch.Tensor) for t in (*dense, out)), view.seq_length, len(view.key_blocks)))
        assert all(torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b for a, b in zip(*results)), step
    assert N.take_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("block,pages,tail,sink", [(16, 5, 7, 4), (64, 0, 3, 3), (64, 3, 0, 4), (256, 2, 100, 0)])
def test_paged_decode_is_that_of_the_general_path(block, pages, tail, sink):
    from inquant.triton_attention import SharedDecodeWorkspace
    from inquant_vllm.kernels import paged_decode
    from inquant_vllm.layout import PageLayout, pack_pages
    heads, q_heads = 4, 28
    layout, workspace = PageLayout(block, heads), SharedDecodeWorkspace()
    pool = torch.zeros((pages + 1, layout.page_bytes), dtype=torch.uint8, device="cuda")
    if pages:
        k, v = (x[0].view(heads, pages, block, 128).transpose(0, 1) for x in workloads.make_kv_torch(6, heads, pages * block, "cuda", 128))
        pool[:pages] = pack_pages(k.to(torch.bfloat16), v.to(torch.bfloat16), layout).view(pages, -1)
    dense = torch.randn((2, heads, block + 4, 128), device="cuda").to(torch.bfloat16)
    ids = torch.randperm(pages, device="cuda")
    query = torch.randn((1, q_heads, 128), device="cuda").to(torch.bfloat16)
    given = torch.empty_like(query)
    outputs = [paged_decode(q, pool, i, dense, pages, tail, sink, layout, workspace, 128 ** -0.5, output=o)
               for q, i, o in ((query, ids.int(), None), (query, ids.int(), given), (query, ids, None), (query.as_subclass(Wrapped), ids.int(), None))]
    assert outputs[1] is given
    assert all(torch.equal(o.as_subclass(torch.Tensor), outputs[0]) for o in outputs)


def test_calls_outside_the_native_path_keep_their_errors():
    from inquant.triton_attention import PackedDecodeState
    from inquant.codec import CodecConfig, quantize
    from inquant.value_codec import quantize_values
    k = _rows(1, 2, 64, torch.bfloat16, "contiguous")
    state = PackedDecodeState([quantize(k, CodecConfig(donor_policy="min_error"))], [quantize_values(k)])
    q, tail = _rows(2, 4, 1, torch.bfloat16, "contiguous"), _rows(3, 2, 5, torch.bfloat16, "contiguous")
    state.decode(q, residual_key=tail, residual_value=tail)
    for query, args, error in ((q[:, :3], {}, "divisible"), (q[:, :1], {}, "divisible"), (q, {"scale": -1.0}, "positive and finite"), (q, {"scale": float("nan")}, "positive and finite"),
                               (q, {"residual_key": tail}, "both be provided"), (q, {"residual_key": tail, "residual_value": tail[:, :, 1:]}, "matching"),
                               (q, {"residual_key": tail.half(), "residual_value": tail.half()}, "match query dtype"),
                               (q, {"sink_key": tail[:, :1], "sink_value": tail[:, :1]}, "KV head count"), (q[0], {}, "query must have shape")):
        with pytest.raises(ValueError, match=error):
            state.decode(query, **args)
    with torch.cuda.stream(torch.cuda.Stream()), pytest.raises(RuntimeError, match="one CUDA stream"):
        state.decode(q)


def test_paged_decode_copies_rows_that_do_not_start_on_16_bytes():
    from inquant.triton_attention import SharedDecodeWorkspace
    from inquant_vllm.kernels import paged_decode
    from inquant_vllm.layout import PageLayout, pack_pages
    heads, q_heads, block = 2, 14, 64
    layout, workspace = PageLayout(block, heads), SharedDecodeWorkspace()
    k, v = (x[0].view(heads, 3, block, 128).transpose(0, 1) for x in workloads.make_kv_torch(7, heads, 3 * block, "cuda", 128))
    pool = pack_pages(k.to(torch.bfloat16), v.to(torch.bfloat16), layout).view(3, -1)
    dense = torch.randn((2, heads, block + 4, 128), device="cuda").to(torch.bfloat16)
    ids, query = torch.arange(3, device="cuda", dtype=torch.int32), torch.randn((1, q_heads, 128), device="cuda").to(torch.bfloat16)

    def off(x):
        buffer = torch.empty(x.numel() + 1, dtype=x.dtype, device="cuda")
        buffer[1:] = x.reshape(-1)
        return buffer[1:].view(x.shape)
    expected, of_query, of_dense = (paged_decode(q, pool, ids, d, 3, 9, 4, layout, workspace, 128 ** -0.5)
                                    for q, d in ((query, dense), (off(query), dense), (query, off(dense))))
    assert torch.equal(of_query, expected) and torch.equal(of_dense, expected)
    with pytest.raises(ValueError, match="start on 16 bytes"):
        paged_decode(query, off(pool), ids, dense, 3, 9, 4, layout, workspace, 128 ** -0.5)


@pytest.mark.parametrize("validate", [False, True])
def test_append_with_the_keywords_of_an_attention_module_is_native(served, validate):
    """The form in which a patched model's attention appends: angles and the position beside the states."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    config = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=16, residual_length=8, sink_tokens=4, value_bits=2,
                         validate_positions=validate)
    prompt, angles = [_rows(s, 2, 30, torch.bfloat16, "contiguous") for s in (1, 2)], torch.zeros(4, device="cuda")
    caches = [InQuantCache(config) for _ in range(2)]
    for cache in caches:
        cache.update(*prompt, 0)
    for step in range(20):      # two seals among them, by tokens that complete a tail in place
        new = [_rows(10 * step + s, 2, 1, torch.bfloat16, "token-major") for s in (3, 4)]
        position = torch.tensor([30 + step], device="cuda")
        views = [cache.append_for_attention(*new, 0, kwargs) for cache, kwargs in
                 zip(caches, (None, {"sin": angles, "cos": angles, "cache_position": position}))]
        assert all(torch.equal(getattr(views[0], n), getattr(views[1], n)) for n in ("sink_key", "sink_value", "residual_key", "residual_value"))
        assert views[0].seq_length == views[1].seq_length == 31 + step
    assert len(served["append_token"]) == 40 and all(served["append_token"])
    wrong = {"cache_position": torch.tensor([3], device="cuda")}
    if validate:
        with pytest.raises(ValueError, match="contiguous append positions"):
            caches[1].append_for_attention(*new, 0, wrong)
        assert len(served["append_token"]) == 40 and caches[1].get_seq_length(0) == 50
    with pytest.raises(ValueError, match="1D integer tensor"):
        caches[1].append_for_attention(*new, 0, {"cache_position": 50})


def test_calls_without_the_native_host_side_give_the_same(monkeypatch):
    """An extension that does not load leaves every call to the Python code."""
    from inquant import _native as N
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.triton_attention import PackedDecodeState, SharedDecodeWorkspace
    from inquant_vllm.kernels import paged_decode
    from inquant_vllm.layout import PageLayout
    config = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=8, sink_tokens=4, value_bits=2)
    layout, dense = PageLayout(64, 2), torch.randn((2, 2, 68, 128), device="cuda").to(torch.bfloat16)
    prompt, query = [_rows(s, 2, 150, torch.bfloat16, "contiguous") for s in (1, 2)], _rows(3, 8, 1, torch.bfloat16, "contiguous")
    new, pool = [_rows(s, 2, 1, torch.bfloat16, "contiguous") for s in (4, 5)], torch.zeros((1, layout.page_bytes), dtype=torch.uint8, device="cuda")

    def run():
        cache = InQuantCache(config)
        cache.update(*prompt, 0)
        view = cache.append_for_attention(*new, 0)
        state = PackedDecodeState(view.key_blocks, view.value_blocks)
        return (view.residual_key, state.decode(query, residual_key=view.residual_key, residual_value=view.residual_value),
                paged_decode(query[:, :, 0], pool, torch.zeros(1, dtype=torch.int32, device="cuda"), dense, 0, 9, 4, layout,
                             SharedDecodeWorkspace(), 128 ** -0.5))
    expected = run()
    monkeypatch.setattr(N, "_host", None)
    monkeypatch.setattr(N, "_host_sought", False, raising=False)
    monkeypatch.setitem(sys.modules, "inquant._host", None)        # an import of it raises ImportError
    with pytest.warns(RuntimeWarning, match="slower Python form"):
        without = run()
    assert all(torch.equal(a, b) for a, b in zip(expected, without))


def test_ordinary_tensors_are_served_and_no_others(served):
    """Which form each call took: without this, both arms of a comparison could be the Python code."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.triton_attention import PackedDecodeState, SharedDecodeWorkspace
    from inquant_vllm.kernels import paged_decode
    from inquant_vllm.layout import PageLayout
    config = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=8, sink_tokens=4, value_bits=2)
    cache = InQuantCache(config)
    cache.update(*(_rows(s, 2, 150, torch.bfloat16, "contiguous") for s in (1, 2)), 0)
    forms = {"contiguous": True, "token-major": True, "slice": True, "unaligned": False}
    for form in forms:
        view = cache.append_for_attention(*(_rows(s, 2, 1, torch.bfloat16, form) for s in (3, 4)), 0)
    cache.append_for_attention(*(_rows(s, 2, 1, torch.bfloat16, "contiguous").as_subclass(Wrapped) for s in (3, 4)), 0)
    # (what the plain call does not serve is offered again behind its checks)
    assert served["append_token"] == [True, True, True, False, False, False, False]
    state = PackedDecodeState(view.key_blocks, view.value_blocks)
    dense = {"residual_key": view.residual_key, "residual_value": view.residual_value}
    for form in forms:
        state.decode(_rows(5, 8, 1, torch.bfloat16, form), **dense)
    assert served["decode"] == list(forms.values())
    state.decode(_rows(5, 8, 1, torch.float32, "contiguous"), **{n: t.float() for n, t in dense.items()})
    assert served["decode"] == [*forms.values(), False]
    state.decode(_rows(5, 8, 1, torch.bfloat16, "contiguous").as_subclass(Wrapped), **dense)
    assert len(served["decode"]) == 5          # (not even asked)
    layout, workspace = PageLayout(64, 2), SharedDecodeWorkspace()
    pool, ids = torch.zeros((2, layout.page_bytes), dtype=torch.uint8, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    rows, query = torch.randn((2, 2, 68, 128), device="cuda").to(torch.bfloat16), _rows(6, 8, 1, torch.bfloat16, "contiguous")[:, :, 0]
    unaligned = _rows(6, 8, 1, torch.bfloat16, "unaligned")[:, :, 0]
    for q, i in ((query, ids), (unaligned, ids), (query, ids.long())):
        paged_decode(q, pool, i, rows, 0, 5, 4, layout, workspace, 128 ** -0.5)
    assert served["paged_decode"] == [True, False, False]


def test_a_refused_call_ties_a_shared_workspace_to_no_stream():
    from inquant.codec import CodecConfig, quantize
    from inquant.triton_attention import PackedDecodeState, SharedDecodeWorkspace
    from inquant.value_codec import quantize_values
    from inquant_vllm.kernels import paged_decode
    from inquant_vllm.layout import PageLayout
    side = torch.cuda.Stream()
    k, q = _rows(1, 2, 64, torch.bfloat16, "contiguous"), _rows(2, 8, 1, torch.bfloat16, "contiguous")
    blocks = [quantize(k, CodecConfig(donor_policy="min_error"))], [quantize_values(k)]
    pool = SharedDecodeWorkspace()
    torch.cuda.synchronize()
    with torch.cuda.stream(side), pytest.raises(ValueError, match="match query dtype"):
        PackedDecodeState(*blocks, workspace_pool=pool).decode(q, residual_key=k.half(), residual_value=k.half())
    torch.cuda.synchronize()
    PackedDecodeState(*blocks, workspace_pool=pool).decode(q, residual_key=k, residual_value=k)
    layout, workspace = PageLayout(64, 2), SharedDecodeWorkspace()
    pages, ids = torch.zeros((1, layout.page_bytes), dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    dense = torch.randn((2, 2, 68, 128), device="cuda").to(torch.bfloat16)

    def paged(query):
        return paged_decode(query[:, :, 0], pages, ids, dense, 0, 9, 4, layout, workspace, 128 ** -0.5)
    torch.cuda.synchronize()
    with torch.cuda.stream(side), pytest.raises(ValueError, match="one BF16 query"):
        paged(q.half())
    paged(q)
    torch.cuda.synchronize()
    with torch.cuda.stream(side), pytest.raises(RuntimeError, match="one CUDA stream"):     # a served call ties it, as before
        paged(q)
