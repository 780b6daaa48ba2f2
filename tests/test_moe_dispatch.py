"""Which of the sparse mixture's two device paths a size takes."""
import pytest

from neuronx_distributed_llama3_2_b200.modules.moe.sparse import pairs_win


# (tokens, width, ff, chosen, shared, gated) and the path that was the faster one in captured graphs, on both sides of the line
@pytest.mark.parametrize("tokens,width,ff,top,shared,gated,pairs", [
    (1, 256, 256, 2, 0, True, True), (64, 256, 256, 2, 0, True, True), (256, 256, 512, 2, 0, True, False), (1, 512, 512, 4, 0, True, False),
    (64, 512, 128, 1, 0, True, True), (1, 1024, 512, 4, 0, True, False), (1, 2048, 64, 1, 0, True, False), (1, 2048, 64, 2, 0, False, True),
    (4, 2048, 512, 2, 0, False, True), (64, 2048, 512, 2, 0, False, False), (64, 1024, 512, 4, 0, True, False),
    (8190, 2048, 2048, 2, 0, True, False)])
def test_small_mixtures_take_the_pairs(tokens, width, ff, top, shared, gated, pairs):
    assert pairs_win(tokens, top, width, ff, shared, gated) is pairs


# the same where one launch sorts the pairs and the router runs in the experts' call
@pytest.mark.parametrize("tokens,width,ff,top,shared,gated,pairs", [
    (1, 512, 128, 1, 0, True, True), (2, 384, 512, 4, 0, True, False), (101, 512, 384, 1, 0, True, False), (4, 768, 384, 2, 0, True, False),
    (6, 768, 512, 1, 512, True, False), (1, 256, 1024, 4, 0, False, False), (28, 384, 768, 2, 0, False, False), (8, 2048, 64, 1, 0, False, True)])
def test_the_line_of_the_single_call(tokens, width, ff, top, shared, gated, pairs):
    assert pairs_win(tokens, top, width, ff, shared, gated) is pairs
