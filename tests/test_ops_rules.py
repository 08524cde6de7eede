"""Launch rules of the Python face of the kernels that are plain arithmetic on a step's shape (no GPU needed)."""
from kvad_b200.ops import Ops


def test_decode_key_ranges_keep_a_launch_one_wave():
    sms = 148
    for heads in (1, 3, 12, 16, 25, 40):
        for rows in list(range(1, 70)) + [128, 500]:
            for table_width in (1, 4, 16, 64):
                s = Ops.decode_splits(rows, heads, table_width, n_sms=sms)
                assert 1 <= s <= min(6, table_width)
                if s > 1:
                    assert s * rows * heads <= 2.75 * sms            # more than one range only while that stays one wave
                if s < min(6, table_width):
                    assert (s + 1) * rows * heads > 2.75 * sms       # and as many ranges as fit it
    # the batch sizes the rule was measured at (12 heads): see Ops.decode_splits
    assert [Ops.decode_splits(r, 12, 16, n_sms=sms) for r in (1, 2, 4, 8, 12, 16, 20, 24, 64)] == [6, 6, 6, 4, 2, 2, 1, 1, 1]
    # it depends on the device's size, not on a constant
    assert Ops.decode_splits(8, 12, 16, n_sms=74) == 2


def test_recurrences_go_in_chunks_by_the_longest_run():
    import torch
    ops = Ops(torch.float32)
    ops.chunked_recurrences = True
    rule = lambda lens, told=True: ops._chunk_rule(sum(lens), len(lens), max(lens) if told else None)          # noqa: E731
    assert rule([1000]) == (True, 0) and rule([300, 300]) == (True, 0)          # nothing short can be beside them
    assert rule([1000] + [1] * 8) == (True, 16)                                  # a prompt among decoding sequences: they keep to the walk
    assert rule([245, 23, 153, 76]) == (True, 16)
    assert rule([159, 159]) == (False, 0) and rule([1] * 2000) == (False, 0)
    # without the longest run: the average, for all sequences alike
    assert rule([1000, 517, 37], told=False) == (True, 0) and rule([1000] + [1] * 8, told=False) == (False, 0)
    ops.chunked_recurrences = False
    assert rule([1000]) == (False, 0)


def test_a_constant_that_chooses_a_kernel_is_part_of_a_captured_step():
    import torch
    ops = Ops(torch.bfloat16)
    for name in ("SPLIT_MIN_ROWS", "SCORED_PROMPT_MIN_NEW", "CHUNK_MIN_ROWS", "CHUNK_SHORT_ROWS", "CHUNK_WORK_BYTES", "SUMS_MIN_K", "ROWS_LINEAR_MAX_OUT",
                 "ROWS_BLOCKS_MAX", "HEADS_LINEAR_MAX_ROWS", "split_linear", "scored_prompt", "chunked_recurrences", "pieces_linear", "scored_wide", "PIECES_MIN_ROWS", "PIECES_MIN_K",
                 "PIECES_WORK_BYTES", "SHORT_PROMPT_KEYS", "SHORT_PROMPT_MAX"):
        before = ops.path_key()
        setattr(ops, name, getattr(ops, name) + 1)
        assert ops.path_key() != before, name
    before = ops.path_key()
    ops.PIECES_ONE_TILE = (256, *ops.PIECES_ONE_TILE[1:])
    assert ops.path_key() != before
