"""Which way the gradient of an embedding goes, on both sides of each line of the rule."""
import pytest

from hetu_galvatron_b200.ops import _lib


# the last count that a sort of 8192 and of 16384 keys is for and one more, tables whose clearing hides the sort and smaller ones, tables
# so large that few tokens save less than they cost, rows that a key does not number, a table that does not start on 16 bytes
@pytest.mark.parametrize("tokens,rows,H,runs", [
    (8192, 32000, 4096, True), (8193, 32000, 4096, False), (8193, 58479, 4096, True), (16384, 32000, 4096, True),
    (16385, 152064, 3584, False), (8192, 19008, 3584, False), (8192, 24576, 4096, True), (4097, 24327, 4096, False),
    (4096, 12288, 4096, True), (4096, 152064, 3584, True), (1024, 152064, 3584, False), (4096, 50304, 1600, True),
    (4096, 50304, 768, False), (1024, 16000, 4096, True), (1024, 3072, 4096, False), (256, 8521, 4096, False),
    (4096, 262143, 4096, True), (4096, 262144, 4096, False)])
def test_rule_of_the_sorted_gradient(tokens, rows, H, runs):
    takes = _lib.load().hg_embedding_bwd_runs_takes
    assert bool(takes(1 << 20, tokens, H, rows)) is runs and not takes((1 << 20) + 8, tokens, H, rows)
