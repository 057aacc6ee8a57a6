"""Chunked-prefill attention (tcgen05 kernel) against float32 causal attention computed by torch
from the same bf16/fp16 tensors, and against the cache's materialising semantics."""
import numpy as np
import pytest
import torch

from helpers import attention_close, to_numpy

pytestmark = pytest.mark.gpu


def _reference(q, k, v, scale):
    """fp32 causal attention; query i sees keys 0 .. L - Tq + i."""
    q32, k32, v32 = q.float(), k.float(), v.float()
    groups = q.shape[1] // k.shape[1]
    k32 = k32.repeat_interleave(groups, dim=1)
    v32 = v32.repeat_interleave(groups, dim=1)
    tq, tk = q.shape[2], k.shape[2]
    s = torch.einsum("bhqd,bhkd->bhqk", q32, k32) * scale
    pos = torch.arange(tq, device=q.device)[:, None] + (tk - tq)
    s = s.masked_fill(torch.arange(tk, device=q.device)[None, :] > pos, float("-inf"))
    return torch.einsum("bhqk,bhkd->bhqd", torch.softmax(s, dim=-1), v32)


@pytest.mark.parametrize("q_heads,kv_heads,q_tokens,history,dtype", [
    (2, 1, 128, 0, torch.bfloat16),        # one tile, pure causal
    (4, 2, 256, 128, torch.bfloat16),      # full tiles with history
    (7, 1, 200, 77, torch.bfloat16),       # ragged query and history lengths, GQA 7
    (4, 4, 1, 300, torch.bfloat16),        # a single query token
    (8, 2, 384, 1000, torch.float16),      # fp16, several KV tiles
    (28, 4, 512, 2048, torch.bfloat16),    # Qwen2.5-7B head counts; items cut into 2 KV segments
    (28, 4, 2048, 6144, torch.bfloat16),   # config 2's chunk shape: 224 items cut into 3 KV segments each
    (3, 1, 300, 5000, torch.float16),      # few items over a long history: cut into 8 segments
    (28, 4, 4224, 0, torch.bfloat16),      # a long unchunked prompt: many items, no cut, ragged last pair
])
def test_prefill_attention_matches_fp32_causal_attention(q_heads, kv_heads, q_tokens, history, dtype):
    from inquant.prefill import prefill_attention
    gen = torch.Generator(device="cuda").manual_seed(11 + q_tokens + history)
    q = torch.randn((1, q_heads, q_tokens, 128), device="cuda", generator=gen).to(dtype)
    k = torch.randn((1, kv_heads, history + q_tokens, 128), device="cuda", generator=gen).to(dtype)
    v = torch.randn((1, kv_heads, history + q_tokens, 128), device="cuda", generator=gen).to(dtype)
    k[:, :, :, 5] *= 6.0   # an outlier channel sharpens the softmax
    scale = 128 ** -0.5
    out = prefill_attention(q, k, v, scale)
    from inquant import _native
    assert _native.take_status(q.device) == 0
    expected = _reference(q, k, v, scale)
    attention_close(to_numpy(out.float())[0], to_numpy(expected)[0])


@pytest.mark.parametrize("q_tokens,history,dtype", [(129, 256, torch.bfloat16), (200, 700, torch.float16), (256, 5000, torch.bfloat16)])
def test_prefill_attention_when_the_maximum_rises_tile_after_tile(q_tokens, history, dtype):
    """Keys with a ramp in one channel, queries of +-8 there, the sign at random from row to row: for about
    half of the rows of every warp each KV tile raises the reference maximum by more than the slack, the
    others keep that of their first tile (both asserted below on the scores).  900 keys are one segment of
    eight tiles, 5256 eight segments of five or six.  Bound: that of bf16 outputs."""
    from inquant.prefill import prefill_attention
    from inquant import _native as N
    tile, slack = 128, 8.0                                      # csrc/prefill.cu: kPfTile, kPfSlack
    gen = torch.Generator(device="cuda").manual_seed(q_tokens)
    q = torch.randn((1, 4, q_tokens, 128), device="cuda", generator=gen)
    q[..., 7] = torch.where(q[..., 7] > 0, 8.0, -8.0)
    q = q.to(dtype)
    k = torch.randn((1, 2, history + q_tokens, 128), device="cuda", generator=gen) * 0.1
    v = torch.randn((1, 2, history + q_tokens, 128), device="cuda", generator=gen).to(dtype)
    k[..., 7] += 16.0 * torch.arange(1, history + q_tokens + 1, device="cuda") / tile   # base-2 scores rise by 16.3 a tile
    k = k.to(dtype)
    scores = q[0].double() @ k[0].double().repeat_interleave(2, 0).transpose(1, 2) * 128 ** -0.5 * 1.4426950408889634
    tops = torch.stack([tile_scores.amax(-1) for tile_scores in scores.split(tile, -1)[:history // tile]], -1)   # tiles that every row sees
    rising = tops.diff(dim=-1).min(-1).values > slack
    assert 0.4 < rising.double().mean() < 0.6 and torch.equal(tops.diff(dim=-1).max(-1).values < 0, ~rising)
    assert all((rows.any(-1) & ~rows.all(-1)).all() for rows in rising[:, :128].split(32, -1))   # both kinds in a warp
    out = prefill_attention(q, k, v, 128 ** -0.5)
    attention_close(to_numpy(out.float())[0], to_numpy(_reference(q, k, v, 128 ** -0.5))[0])
    assert N.take_status(q.device) == 0


def test_prefill_attention_accepts_strided_views_and_rejects_bad_arguments():
    from inquant.prefill import prefill_attention
    gen = torch.Generator(device="cuda").manual_seed(3)
    # [1, T, H, D] projections viewed as [1, H, T, D], as a model produces them
    q = torch.randn((1, 160, 4, 128), device="cuda", generator=gen).bfloat16().transpose(1, 2)
    k = torch.randn((1, 400, 2, 128), device="cuda", generator=gen).bfloat16().transpose(1, 2)
    v = torch.randn((1, 400, 2, 128), device="cuda", generator=gen).bfloat16().transpose(1, 2)
    out = prefill_attention(q, k, v, 0.1)
    attention_close(to_numpy(out.float())[0], to_numpy(_reference(q, k, v, 0.1))[0])
    with pytest.raises(ValueError):
        prefill_attention(q, k[:, :, :100], v[:, :, :100])          # fewer keys than queries
    with pytest.raises(NotImplementedError):
        prefill_attention(q.float(), k.float(), v.float())
    with pytest.raises(ValueError):
        prefill_attention(q[:, :3], k, v)                            # 3 query heads over 2 KV heads


def test_prefill_chunks_through_the_cache_match_one_shot_attention_over_materialised_history():
    """16 chunks... here 3 chunks of 256: every chunk attends to the cache's dequantised history
    plus itself, exactly what `InQuantCache.update` hands to the model's attention."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.prefill import prefill_chunk
    gen = torch.Generator(device="cuda").manual_seed(19)
    heads, q_heads, chunk, chunks = 2, 14, 256, 3
    cfg = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=16, sink_tokens=4,
                      value_bits=2, value_group_size=64)
    cache, shadow = InQuantCache(cfg), InQuantCache(cfg)
    scale = 128 ** -0.5
    for c in range(chunks):
        q = torch.randn((1, q_heads, chunk, 128), device="cuda", generator=gen).bfloat16()
        k = torch.randn((1, heads, chunk, 128), device="cuda", generator=gen).bfloat16()
        v = torch.randn((1, heads, chunk, 128), device="cuda", generator=gen).bfloat16()
        out = prefill_chunk(cache, q, k, v, 0, scale)
        full_k, full_v = shadow.update(k, v, 0)
        assert full_k.shape[2] == (c + 1) * chunk
        attention_close(to_numpy(out.float())[0], to_numpy(_reference(q, full_k, full_v, scale))[0])
    for a, b in zip(cache.materialize(0), shadow.materialize(0)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("value_bits,chunk_sizes", [(2, (256, 256, 256, 100, 37)), (None, (300, 212)), (4, (64, 1, 500))])
def test_prefill_history_holds_exactly_what_update_would_return(value_bits, chunk_sizes):
    """The dense history kept across chunks is bit-identical to the tensors `InQuantCache.update`
    rebuilds per chunk, so the two forms of `prefill_chunk` give the same attention, and both caches
    end up with the same contents."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.prefill import PrefillHistory, prefill_chunk
    gen = torch.Generator(device="cuda").manual_seed(23)
    heads, q_heads = 2, 14
    cfg = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=16, sink_tokens=4,
                      value_bits=value_bits, value_group_size=64)
    cache, shadow, plain = InQuantCache(cfg), InQuantCache(cfg), InQuantCache(cfg)
    history = PrefillHistory(cache, capacity_tokens=128, persistent=True)      # forces the tensors to grow
    scale, seen = 128 ** -0.5, 0
    for tokens in chunk_sizes:
        q = torch.randn((1, q_heads, tokens, 128), device="cuda", generator=gen).bfloat16()
        k = torch.randn((1, heads, tokens, 128), device="cuda", generator=gen).bfloat16()
        v = torch.randn((1, heads, tokens, 128), device="cuda", generator=gen).bfloat16()
        out = prefill_chunk(cache, q, k, v, 0, scale, history=history)
        full_k, full_v = shadow.update(k, v, 0)
        seen += tokens
        key, value = history._layers[0][0], history._layers[0][1]
        assert history._layers[0][2] == seen == cache.get_seq_length(0)
        assert torch.equal(out, prefill_chunk(plain, q, k, v, 0, scale))
        attention_close(to_numpy(out.float())[0], to_numpy(_reference(q, full_k, full_v, scale))[0])
        # after sealing, the history equals what the NEXT update would put before its new states
        next_k, next_v = shadow.materialize(0)
        assert torch.equal(key[:, :, :seen], next_k) and torch.equal(value[:, :, :seen], next_v)
    for a, b in zip(cache.materialize(0), shadow.materialize(0)):
        assert torch.equal(a, b)
    assert history.nbytes > 0
    # a history first used on a filled layer takes the dense state over from the cache
    late = PrefillHistory(plain, persistent=True)
    q = torch.randn((1, q_heads, 50, 128), device="cuda", generator=gen).bfloat16()
    k = torch.randn((1, heads, 50, 128), device="cuda", generator=gen).bfloat16()
    assert torch.equal(prefill_chunk(plain, q, k, k, 0, scale, history=late), prefill_chunk(cache, q, k, k, 0, scale, history=history))
    seen += 50
    # an update behind the history's back is detected
    k = torch.randn((1, heads, 8, 128), device="cuda", generator=gen).bfloat16()
    cache.update(k, k, 0)
    with pytest.raises(RuntimeError, match="state mismatch"):
        prefill_chunk(cache, torch.zeros((1, q_heads, 8, 128), device="cuda", dtype=torch.bfloat16), k, k, 0, scale, history=history)
    with pytest.raises(ValueError, match="another cache"):
        prefill_chunk(plain, torch.zeros((1, q_heads, 8, 128), device="cuda", dtype=torch.bfloat16), k, k, 0, scale, history=history)
    history.release()
    assert history.nbytes == 0


def test_prefill_history_reports_non_finite_input_at_check_or_at_once():
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.prefill import PrefillHistory, prefill_chunk
    cfg = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=16, sink_tokens=4, value_bits=2)
    q = torch.zeros((1, 4, 200, 128), device="cuda", dtype=torch.bfloat16)
    k = torch.randn((1, 2, 200, 128), device="cuda").bfloat16()
    bad = k.clone()
    bad[0, 1, 30, 7] = float("inf")
    cache = InQuantCache(cfg)
    history = PrefillHistory(cache)
    prefill_chunk(cache, q, k, k, 0, history=history)
    history.check()                                  # nothing to report
    prefill_chunk(cache, q, bad, k, 0, history=history)   # deferred: no exception here
    with pytest.raises(ValueError, match="finite"):
        history.check()
    history.check()                                  # the report clears the word
    strict = InQuantCache(cfg)
    with pytest.raises(ValueError, match="finite"):
        prefill_chunk(strict, q, bad, k, 0, history=PrefillHistory(strict, defer_checks=False))


def test_prefill_history_without_a_dense_copy_rebuilds_from_the_packed_cache():
    """The default history keeps no per-layer dense tensors: every chunk's history comes out of the
    packed cache into one scratch pair shared by the layers.  Outputs and cache contents equal the
    materialising form chunk by chunk, for two layers that alternate."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.prefill import PrefillHistory, prefill_chunk
    gen = torch.Generator(device="cuda").manual_seed(29)
    heads, q_heads = 2, 14
    cfg = CacheConfig(CodecConfig(donor_policy="min_error"), block_size=64, residual_length=16, sink_tokens=4, value_bits=2)
    cache, plain = InQuantCache(cfg), InQuantCache(cfg)
    history = PrefillHistory(cache, capacity_tokens=64)
    assert not history.persistent
    scale = 128 ** -0.5
    for tokens in (3, 200, 130, 70):
        for layer in (0, 1):
            q = torch.randn((1, q_heads, tokens, 128), device="cuda", generator=gen).bfloat16()
            k = torch.randn((1, heads, tokens, 128), device="cuda", generator=gen).bfloat16()
            v = torch.randn((1, heads, tokens, 128), device="cuda", generator=gen).bfloat16()
            out = prefill_chunk(cache, q, k, v, layer, scale, history=history)
            assert torch.equal(out, prefill_chunk(plain, q, k, v, layer, scale))
    history.check()
    for layer in (0, 1):
        for a, b in zip(cache.materialize(layer), plain.materialize(layer)):
            assert torch.equal(a, b)
    assert not history._layers
    assert 0 < history.nbytes <= 2 * heads * 1024 * 128 * 2     # one pair for both layers, grown geometrically
    history.release()
    assert history.nbytes == 0


@pytest.mark.parametrize("q_heads,kv_heads,q_tokens,kv_tokens", [(4, 2, 96, 96), (28, 4, 256, 2048), (28, 4, 1100, 1100)])   # one item per head, cut items with a merge, several rounds
@pytest.mark.parametrize("captured", [False, True])
def test_launches_in_a_row_read_what_the_one_before_wrote(q_heads, kv_heads, q_tokens, kv_tokens, captured):
    """A launch is set up while the one before it runs: every pass reads the output of the pass before it as its
    queries, inputs that a copy has just written, and writes over inputs that the pass before it read."""
    from inquant.prefill import prefill_attention
    gen = torch.Generator(device="cuda").manual_seed(q_tokens)
    start, k0, v0 = (torch.randn((1, h, t, 128), device="cuda", generator=gen).to(torch.bfloat16)
                     for h, t in ((q_heads, q_tokens), (kv_heads, kv_tokens), (kv_heads, kv_tokens)))
    q, k, v = torch.empty_like(start), torch.empty_like(k0), torch.empty_like(v0)

    def chain(settle):
        q.copy_(start), k.copy_(k0), v.copy_(v0)
        for i in range(6):
            settle()
            out = prefill_attention(q, k, v)
            settle()
            prefill_attention(out, k, v, out=q)      # writes what the pass before it read
            settle()
            if i % 2:
                k.mul_(-1.0)
                settle()
        return q

    expected = chain(torch.cuda.synchronize).clone()
    if captured:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            chain(lambda: None)
        graph.replay()
    else:
        chain(lambda: None)
    torch.cuda.synchronize()
    assert torch.isfinite(expected.float()).all() and torch.equal(q, expected)


@pytest.fixture
def restores(monkeypatch):
    """Calls of the two restore entry points: the runs given to one, the blocks given to the other."""
    from inquant import _native as N
    lib, calls = N.library(), []
    history, table = lib.inq_restore_history, lib.inq_restore_blocks_table

    def of_runs(args, stream):
        calls.append(("runs", args._obj.n_runs))
        return history(args, stream)

    def of_blocks(*args):
        calls.append(("blocks", args[2]))
        return table(*args)
    monkeypatch.setattr(lib, "inq_restore_history", of_runs)
    monkeypatch.setattr(lib, "inq_restore_blocks_table", of_blocks)
    return calls


@pytest.mark.parametrize("seals", [32, 33, 70])
def test_history_of_many_seals_is_restored_by_two_launches(restores, seals):
    """A layer sealed block by block: up to 32 runs travel as records, more are addressed through decode descriptors."""
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    from inquant.prefill import PrefillHistory
    gen, heads = torch.Generator(device="cuda").manual_seed(seals), 2
    cache = InQuantCache(CacheConfig(CodecConfig(donor_policy="min_error"), block_size=16, residual_length=8, sink_tokens=4, value_bits=2))

    def states(tokens, n=heads):
        return torch.randn((1, n, tokens, 128), device="cuda", generator=gen).bfloat16()
    cache.update(states(12), states(12), 0)
    for _ in range(seals):
        cache.extend(states(16), states(16), 0)
    assert len(cache._layers[0].runs) == seals
    history = PrefillHistory(cache)
    for tokens, kept in ((3, seals), (16, seals), (5, seals + 1)):       # the second chunk seals a block more
        del restores[:]
        history.chunk(states(tokens, 4), states(tokens), states(tokens), 0)
        assert restores == ([("runs", kept)] if kept <= 32 else [("runs", 0), ("blocks", kept)])
    history.check()
    history.release()
    assert not history._descriptors


@pytest.mark.parametrize("block,fraction", [(256, 0.125), (64, 0.0), (40, 0.25), (16, 0.5), (104, 0.125)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_blocks_restored_through_descriptors_equal_their_own_tensors(restores, monkeypatch, block, fraction, dtype):
    """Blocks that are not whole steps of 16 or parts of 64 tokens, no, 16, 32 and 64 salient channels, blocks of one
    and of several to an encoder launch, beside the dense rows; a layer that was reset starts anew."""
    import inquant.prefill as prefill
    from inquant.cache import CacheConfig, InQuantCache
    from inquant.codec import CodecConfig
    monkeypatch.setattr(prefill, "_TABLE_RUNS", 1)
    gen, heads = torch.Generator(device="cuda").manual_seed(block), 3
    cache = InQuantCache(CacheConfig(CodecConfig(donor_policy="min_error", salient_fraction=fraction), block_size=block,
                                     residual_length=8, sink_tokens=4, value_bits=2))
    history = prefill.PrefillHistory(cache)

    def states(tokens, n=heads):
        return torch.randn((1, n, tokens, 128), device="cuda", generator=gen).to(dtype)
    for _ in range(2):
        for step, tokens in enumerate((20, 3 * block, 1, block + 3, 2 * block, 7, block)):
            key, value = states(tokens), states(tokens)
            layer = cache._layers.get(0)
            expected = (key, value) if layer is None else [
                torch.cat([sink, *(b.dequantize() for b in blocks), tail, new], dim=2) for sink, blocks, tail, new in
                ((layer.sink_key, layer.key_blocks, layer.residual_key, key), (layer.sink_value, layer.value_blocks, layer.residual_value, value))]
            by_table = layer is not None and len(layer.runs) > 1
            del restores[:]
            out = history.chunk(states(tokens, 6), key, value, 0)
            assert ("blocks" in dict(restores)) == by_table and torch.isfinite(out.float()).all()
            for scratch, rows in zip(history._scratch, expected):
                assert torch.equal(scratch[:, :, :rows.shape[2]], rows), (step, tokens)
        assert by_table
        cache.reset()
    history.check()
