"""Prompt attention whose keys are shared out over a cluster: few row tiles behind long and short contexts, blocks without keys."""
import pytest

from test_attn_prefill_gpu import run_case

pytestmark = pytest.mark.gpu


# head dim, first chunk, second chunk, sequences, heads: 2, 4 and 8 splits; more splits than key tiles; a ragged last row tile
@pytest.mark.parametrize("hd,T1,T2,B,H", [(64, 700, 123, 1, 32), (128, 300, 33, 1, 16), (64, 1500, 40, 1, 3), (128, 32, 1000, 1, 2), (64, 64, 900, 2, 2), (128, 600, 65, 3, 12)])
def test_splits(hd, T1, T2, B, H):
    assert run_case(hd, T1, T2, B, H) <= 2e-5        # the bound of the single-block form


# a cache far larger than the keys: blocks of a cluster that leave, those that share two tiles and more (one tile, fewer and more tiles than blocks), four blocks at most
@pytest.mark.parametrize("hd,T1,T2,B,H", [(64, 32, 33, 1, 2), (128, 32, 64, 1, 16), (128, 33, 32, 2, 12), (64, 100, 130, 1, 8), (128, 64, 200, 1, 1)])
def test_splits_by_the_keys(hd, T1, T2, B, H):
    assert run_case(hd, T1, T2, B, H, spare=4000) <= 2e-5
