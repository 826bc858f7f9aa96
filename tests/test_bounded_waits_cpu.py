"""A kernel whose wait for the copy engine gave up stops before it writes anything of that tile.  A lost copy cannot be brought
about on a GPU, so this reads the source: the warp-owned kernel A does not vote at the wait, where it would cost every tile a barrier,
but at the next barrier of each way to its outputs."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, '..', 'ista-daslab-optimizers_b200', 'csrc')
VOTE = 'if (__syncthreads_or(lost)) return;'


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r'//[^\n]*', '', re.sub(r'/\*.*?\*/', '', text, flags=re.S))


def _braces(text, at):
    """The text between the brace at or behind `at` and its partner, and where it ends."""
    start = text.index('{', at)
    depth = 0
    for i in range(start, len(text)):
        depth += {'{': 1, '}': -1}.get(text[i], 0)
        if depth == 0:
            return text[start + 1:i], i + 1
    raise AssertionError('unbalanced braces')


def test_every_wait_votes_before_outputs():
    for name in ('ef_topk_quant.cu', 'ef_topk_quant_bf16.cu', 'ef_topk_quant_f32.cu', 'window_adam.cu'):
        waits = re.findall(r'mbar_wait\(&s_bar[^;]*;(.*?)\{(.*?)\}', _source(name), flags=re.S)
        assert waits, name
        for between, then in waits:
            assert between.split('if')[-1].strip() == '(__syncthreads_or(!ok))', name
            assert 'return;' in then, name


def test_warp_owned_tiles_vote_on_every_way_to_their_outputs():
    text = _source('ef_topk_quant_bf16_warps.cu')
    kernel = text[text.index('ef_topk_quant_bf16_warps_kernel('):]
    tile, _ = _braces(kernel, kernel.index('for (int unit = unit0'))
    wait, chosen = tile.index('mbar_wait('), tile.index('if (ok) {')
    for output in ('i_out', 'v_out', 'qe[', 'stats_encode', 'residual_and_extremes', 'select_by_bisection', 'select_from_units', 'atomicMin'):
        assert output not in tile[wait:chosen], output
    attempts, _ = _braces(tile, tile.index('for (int attempt'))
    assert attempts.count('ok = true') == 1 and tile[wait:chosen].count('ok = true') == 1
    assert VOTE in attempts[:attempts.index('ok = true')]
    _, end = _braces(tile, chosen)
    other, _ = _braces(tile, tile.index('else', end))
    assert other.strip().startswith(VOTE)
