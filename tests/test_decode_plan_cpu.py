"""Host side of a decode launch: the work list of uneven batches against the merge scratch (no GPU)."""
import ctypes

import pytest

from inquant import _native as N


def _shape(starts, block_tokens, n_pad, ctas_per_sm, value_kind=0, value_groups=2):
    shape = N.DecodeShape()
    rc = N.library().inq_decode_launch_shape(len(starts) - 1, starts[-1], block_tokens, n_pad, value_kind, value_groups, ctas_per_sm,
                                             ctypes.byref(shape))
    assert rc == N.OK
    return shape


def _most_parts(starts, shape):
    """Largest number of CTA ranges that hold slices of one pair, by the kernel's own arithmetic."""
    most = 0
    for pair in range(len(starts) - 1):
        lo, hi = (starts[pair + k] + (pair + 1) * shape.ramp_units for k in (0, 1))
        most = max(most, (hi - 1) // shape.per_cta - lo // shape.per_cta + 1)
    return most


def _batches(block_tokens):
    """Slices per pair: even batches, one long sequence among short ones, one pair alone, heads of a layer."""
    per_block = max(1, block_tokens // 32)
    for heads in (1, 2, 8):
        for long, others in ((5000, 15), (8000, 15), (40000, 63), (600, 3), (5000, 0), (1, 300)):
            for position in {0, others // 2, others}:
                units = [long * per_block if i == position else per_block for i in range(others + 1)]
                starts = [0]
                for u in units:
                    for _ in range(heads):
                        starts.append(starts[-1] + u)
                yield starts


@pytest.mark.parametrize("block_tokens", [16, 64, 256])
@pytest.mark.parametrize("n_pad", [0, 1, 16, 17, 32, 48, 64])
def test_merge_of_the_most_divided_pair_fits_the_shared_memory_of_the_launch(block_tokens, n_pad):
    for ctas_per_sm in (1, 2, 3, 4):
        for starts in _batches(block_tokens):
            shape = _shape(starts, block_tokens, n_pad, ctas_per_sm)
            total = starts[-1] + (len(starts) - 1) * shape.ramp_units
            assert (shape.n_ctas - 1) * shape.per_cta < total <= shape.n_ctas * shape.per_cta
            assert _most_parts(starts, shape) <= shape.merge_parts, (starts[-1], len(starts) - 1, ctas_per_sm)
            assert shape.shared_bytes <= 227 * 1024
            assert (shape.n_ctas + len(starts) - 1) * N.RECORD_FLOATS <= N.library().inq_decode_workspace_floats(len(starts) - 1, starts[-1])


@pytest.mark.parametrize("value_kind,value_groups", [(1, 0), (2, 1), (2, 2), (2, 4), (0, 1), (0, 4)])
def test_merge_fits_with_the_other_value_codecs(value_kind, value_groups):
    for starts in _batches(64):
        shape = _shape(starts, 64, 16, 3, value_kind, value_groups)
        assert _most_parts(starts, shape) <= shape.merge_parts


def test_a_long_request_beside_short_ones_takes_more_parts_than_the_warps_scratch_holds():
    """16-token blocks without salient channels, one KV head, 80000 tokens beside fifteen requests of one
    block: four CTAs per SM give the long pair 556 parts, and the four warps' own 32256 bytes hold 503."""
    starts = [0, 5000] + [5000 + i for i in range(1, 16)]
    shape = _shape(starts, 16, 0, 4)
    assert _most_parts(starts, shape) > 503
    assert shape.merge_parts >= shape.n_ctas


@pytest.mark.parametrize("pairs,units", [(8, 512), (8, 2048), (8, 1024), (16, 4096 // 16)])
def test_four_ctas_per_sm_fill_every_sm_or_leave_the_fourth_out(pairs, units):
    """16-token blocks, a batch whose pairs or work do not give four ranges to all of 148 SMs."""
    starts = [p * units for p in range(pairs + 1)]
    four, three = _shape(starts, 16, 16, 4), _shape(starts, 16, 16, 3)
    assert four.n_ctas == three.n_ctas <= 444 and four.per_cta == three.per_cta
    long = [p * 4096 for p in range(65)]
    assert 444 < _shape(long, 16, 16, 4).n_ctas <= 592


def test_launch_shape_refuses_what_no_launch_could_have():
    lib, shape = N.library(), N.DecodeShape()
    assert lib.inq_decode_launch_shape(1, 1, 16, 0, 0, 2, 4, None) == N.ERR_ARGUMENT
    for bad in ((0, 1, 16, 0, 0, 2, 4), (2, 1, 16, 0, 0, 2, 4), (1, 1, 0, 0, 0, 2, 4), (1, 1, 16, 65, 0, 2, 4), (1, 1, 16, 0, 0, 2, 0)):
        assert lib.inq_decode_launch_shape(*bad, ctypes.byref(shape)) == N.ERR_ARGUMENT


@pytest.mark.parametrize("block_tokens,n_pad", [(16, 16), (64, 16), (256, 16), (16, 48), (40, 0)])
def test_pairs_of_equal_length_are_covered_once_by_resident_ranges(block_tokens, n_pad):
    """The launch without a list of starts, walked as the kernel walks it: every slice of every pair in one range, each
    part with a record of its own inside the workspace, no more parts than the merge's scratch holds."""
    lib, shape = N.library(), N.DecodeShape()
    own = 0
    for ctas_per_sm in (1, 2, 3, 4):
        for pairs in (1, 2, 8, 16, 28 * 4, 32 * 8, 444, 445, 1000):
            for units in (1, 2, 7, 8, 9, 31, 40, 63, 64, 65, 128, 250, 512, 1000, 4096):
                if pairs * units > 200000:
                    continue
                assert lib.inq_decode_launch_shape_uniform(pairs, units, block_tokens, n_pad, 0, 2, ctas_per_sm, ctypes.byref(shape)) == N.OK
                ramp, per, total = shape.ramp_units, shape.per_cta, pairs * (units + shape.ramp_units)
                assert shape.n_ctas <= 148 * ctas_per_sm and (shape.n_ctas - 1) * per < total <= shape.n_ctas * per
                own += ramp + units == per * -(-units // per) and pairs > 1
                workspace = lib.inq_decode_workspace_floats(pairs, pairs * units) // N.RECORD_FLOATS
                ends, parts, records = [0] * pairs, [0] * pairs, set()
                for cta in range(shape.n_ctas):
                    pos, stop = cta * per, min((cta + 1) * per, total)
                    pair = pos // (units + ramp)
                    while pos < stop:
                        first = pair * (units + ramp) + ramp                 # the pair's first slice
                        lo, hi = max(pos, first) - first, min(stop, first + units) - first
                        pos = min(stop, first + units)
                        if hi > lo:
                            assert lo == ends[pair] and cta - first // per == parts[pair]
                            ends[pair], parts[pair] = hi, parts[pair] + 1
                            records.add(cta + pair)
                        pair += 1
                assert ends == [units] * pairs and len(records) == sum(parts) and max(records) < workspace
                assert parts == [(first + units - 1) // per - first // per + 1 for first in (p * (units + ramp) + ramp for p in range(pairs))]
                assert max(parts) <= shape.merge_parts
    assert own > 20      # ranges of their own are among them


def test_uniform_launch_shape_refuses_what_no_launch_could_have():
    lib, shape = N.library(), N.DecodeShape()
    for bad in ((0, 1, 16, 0, 0, 2, 4), (2, 0, 16, 0, 0, 2, 4), (1, 1, 0, 0, 0, 2, 4), (1, 1, 16, 65, 0, 2, 4), (1, 1, 16, 0, 0, 2, 0)):
        assert lib.inq_decode_launch_shape_uniform(*bad, ctypes.byref(shape)) == N.ERR_ARGUMENT
