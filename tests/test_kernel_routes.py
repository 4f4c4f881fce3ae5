"""Which form of a kernel a call takes: the rules of the launchers, without a GPU."""

import pytest
import torch

from ondeviceinfer_b200.kernels import ops


@pytest.mark.parametrize("heads,M,N,K,tile", [
    (16, 1, 512, 64, 8), (16, 8, 256, 96, 8), (16, 9, 512, 64, 16), (16, 100, 256, 64, 16), (16, 100, 512, 128, 16),
    (16, 500, 256, 64, 64), (16, 2048, 512, 64, 64), (16, 500, 512, 128, 64), (16, 500, 256, 96, 64),      # blocks of 16 x 16 outputs do too little
    (16, 2048, 64, 256, 16), (16, 2048, 128, 512, 16), (4, 2048, 72, 40, 16)])
def test_products_per_head_of_many_rows_and_few_k_go_in_tiles_of_64(heads, M, N, K, tile):
    assert ops.grouped_heads_tile(heads, M, N, K) == tile


def test_only_bfloat16_takes_runs_in_chunks():
    floats = lambda least: 7 if least is None else 100 + least
    assert [ops.chunk_floats(None, dtype, floats) for dtype in (torch.bfloat16, torch.float32)] == [7, 0]
    assert ops.chunk_floats(True, torch.float32, floats) == 101 and ops.chunk_floats(False, torch.bfloat16, floats) == 0


@pytest.mark.parametrize("heads,d,lens,chunks", [
    (16, 128, [2048], True), (16, 128, [333, 769, 1777], True), (16, 128, [1000, 1000], True), (16, 128, [1000, 500, 250], True),
    (16, 128, [1000] * 3, False), (16, 128, [512] * 4, False), (16, 128, [200] * 4, False), (32, 128, [256, 256], False),
    (32, 128, [1000, 500], False), (32, 128, [800], True), (8, 128, [512] * 4, True),      # heads of 128: the longest run's chain
    (16, 64, [512] * 4, True), (32, 64, [256, 256], True), (16, 64, [512] * 5, False), (16, 64, [223], False), (4, 128, [224], True), (16, 96, [2048], False)])
def test_head_delta_goes_in_chunks_where_a_run_is_what_the_step_waits_for(heads, d, lens, chunks):
    assert (ops.head_delta_chunk_floats(sum(lens), len(lens), max(lens), heads, d, d) > 0) == chunks


def test_operands_off_the_16_byte_borders_keep_the_tiles_of_the_cuda_cores():
    whole = torch.zeros(65, dtype=torch.bfloat16)
    aligned, off = whole[:64], whole[1:]
    assert aligned.data_ptr() % 16 == 0
    ok = lambda *operands: ops.grouped_tensor_ok((64, 8), torch.bfloat16, *operands)
    assert ok() and ok(aligned, aligned) and not ok(aligned, off)
    assert not ops.grouped_tensor_ok((64, 12), torch.bfloat16, aligned) and not ops.grouped_tensor_ok((64, 8), torch.float32)
    few = ops.grouped_few_rows_ok((64, 8), torch.bfloat16)      # the form for few rows is float32's
    tiles = lambda pairs, *operands: ops.RoutingTable(pairs, 1, 2, "cpu", few_rows_ok=few, tensor=ok(*operands)).tm
    assert [tiles(n, aligned) for n in (2, 16, 17, 100)] == [8, 8, 16, 16] and [tiles(n, off) for n in (2, 16, 64, 65, 100)] == [16, 16, 16, 64, 64]
    assert ops.RoutingTable(2, 1, 2, "cpu", few_rows_ok=ops.grouped_few_rows_ok((64, 8), torch.float32)).tm == 4


@pytest.mark.parametrize("P,N,lens,chunks", [
    (64, 128, [2048], True), (64, 128, [1023], False), (64, 128, [128] * 8, True), (64, 128, [127] * 9, False),
    (32, 256, [130] * 8, False), (20, 64, [130] * 8, False), (32, 256, [256] * 8, True), (32, 256, [1100], True),      # padded to 64 columns
    (64, 48, [2048], False), (6, 64, [2048], False)])
def test_state_space_scan_goes_in_chunks_from_the_runs_that_win_by_it(P, N, lens, chunks):
    assert (ops.ssd_chunk_floats(sum(lens), len(lens), 16, P, N, 1) > 0) == chunks
