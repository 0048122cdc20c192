"""Rules that the bounded waits of the tensor-core kernels keep, read from their source: what happens when a wait runs out
cannot be tried on a GPU without leaving copies in flight behind."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / 'deepep_b200' / 'csrc' / 'kernels'
LANE_ROLES = ('mma_role', 'mma_role_pair')       # functions that one lane runs


def _calls(text):
    """(name, line, opening lines of the blocks around it, the line) of every wait of a pipeline."""
    stack, out = [], []
    text = re.sub(r'//[^\n]*', '', text)
    for number, line in enumerate(text.split('\n'), 1):
        for token in re.finditer(r'\bpipe_wait(?:_lane|_warp)?\(|[{}]', line):
            if token.group() == '{':
                stack.append(line)
            elif token.group() == '}':
                stack.pop()
            else:
                out.append((token.group()[:-1], number, list(stack) + [line[:token.start()]], line))
    return out


@pytest.mark.parametrize('name', ['gemm_sm100.cu', 'tp_fused.cu'])
def test_a_warp_gives_up_as_a_whole(name):
    """One lane may leave on its own only in a role that a single lane runs. Where the whole warp goes on to elect.sync, to
    tensor-memory accesses or to a barrier, its lanes leave together, by a vote: those that stayed would wait without a limit."""
    text = (KERNELS / name).read_text()
    calls = _calls(text)
    assert len(calls) >= 6
    functions = [(m.start(), m.group(1)) for m in re.finditer(r'__device__[^;{]*?\b(\w+)\([^;{]*\{', text)]
    starts = [text.count('\n', 0, at) + 1 for at, _ in functions]
    for kind, line, around, source in calls:
        single = any('lane == 0' in opening for opening in around)
        enclosing = [f for at, (_, f) in zip(starts, functions) if at <= line][-1:]
        single = single or enclosing == [e for e in enclosing if e in LANE_ROLES] != []
        if single:
            assert kind == 'pipe_wait', f'{name}:{line}'
        else:
            assert kind != 'pipe_wait' or 'pipe_alive_warp(pipe_wait(' in source, f'{name}:{line}'
            if kind == 'pipe_wait_lane':        # (nothing is decided by the lane)
                assert not re.search(r'\b(break|return|if)\b', re.sub(r'if constexpr \(!?kFp8\)', '', source)), f'{name}:{line}'
            if kind == 'pipe_wait_warp':        # what it is told to be `seen` has to be the warp's answer as well
                seen = re.search(r'pipe_wait_warp\(pc, (\w+),', source).group(1)
                assert f'{seen} = pipe_test_warp(' in text or f'{seen} = kFp8 ? pipe_test_warp(' in text, f'{name}:{line}'
    for role in LANE_ROLES:
        for call in re.finditer(r'^.*\b%s<.*\(pc.*$' % role, text, re.M):
            assert 'lane == 0' in call.group(), call.group()


def test_scale_warps_meet_also_when_one_has_given_up():
    """The barrier of the scale warps is counted: a warp that leaves before it would keep the others there for good."""
    text = (KERNELS / 'gemm_sm100.cu').read_text()
    assert 'bar.sync 3' not in text and text.count('ok = sf_barrier(ok);') == 2 and text.count('sf_barrier(true);') == 2
