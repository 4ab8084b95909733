"""CPU: no kernel of a dependent chain may end before it has waited for the grid in front.

The kernels of a call are launched as programmatic dependents (``launch_after``).  A grid that completes without having waited
lets what follows on the stream start while the grid in front still writes, so every way out of such a kernel lies behind
``grid_dep_wait()``.  Two kernels wait late and have ways out in front of that; a way out that only an expired wait takes is not
one that a run shows, so the rule is checked on the source.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'nha_b200', 'csrc')


def _source(path):
    text = open(path).read()
    text = re.sub(r'/\*.*?\*/', ' ', text, flags=re.S)
    text = re.sub(r'//[^\n]*', '', text)
    return re.sub(r'^[ \t]*#(?:[^\n]*\\\n)*[^\n]*', '', text, flags=re.M)     # directives, macro bodies among them


SOURCES = {os.path.basename(p): _source(p) for p in sorted(glob.glob(os.path.join(CSRC, '*.cu')))}


def _block(text, at):
    """The block that opens at text[at], braces included."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == '{') - (text[i] == '}')
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError('unbalanced braces')


def _body(text, kernel):
    m = re.search(r'__global__[^;{]*?\b' + kernel + r'\s*\(', text)
    return _block(text, text.index('{', m.end())) if m else None


def ways_out_without_wait(body):
    """The `return`s of a kernel's body, and its end, that no grid_dep_wait() precedes on every path to them.  A wait counts for the
    block it stands in and the blocks inside that, and for the block around it where a named warp does it: the grid has not completed
    while that warp waits."""
    bad, blocks, start = [], [], 0
    for m in re.finditer(r'[;{}]', body):
        i, c = m.start(), m.group()
        text = ' '.join(body[start:i].split())
        start = i + 1
        if c == '{':
            blocks.append({'head': text, 'waited': False, 'lambda': bool(re.search(r'=\s*\[[&=]\]', text))})
        elif c == '}':
            b = blocks.pop()
            if not blocks:
                if not b['waited']:
                    bad.append('end of the kernel')
            elif b['waited'] and re.fullmatch(r'if \(warp == \d+\)', b['head']):
                blocks[-1]['waited'] = True
        elif text == 'grid_dep_wait()':
            blocks[-1]['waited'] = True
        elif re.search(r'\breturn$', text) and not any(b['lambda'] for b in blocks) and not any(b['waited'] for b in blocks):
            bad.append(text + ' in ' + (blocks[-1]['head'] or 'the kernel'))
    return bad


def _dependent_kernels():
    launched = {k for t in SOURCES.values() for k in re.findall(r'launch_after\((nha_\w+)', t)}
    kernels = {k for t in SOURCES.values() for k in re.findall(r'__global__[^;{]*?\b(nha_\w+_kernel)\s*\(', t)}
    chained = {k for k in kernels for t in SOURCES.values() if 'grid_dep_launch()' in (_body(t, k) or '')}
    return sorted((launched | chained) - {'nha_decode_stream_kernel'})     # (which may be launched without the attribute: nothing to wait for)


@pytest.mark.parametrize('kernel', _dependent_kernels())
def test_every_way_out_lies_behind_the_wait(kernel):
    bodies = [b for b in (_body(t, kernel) for t in SOURCES.values()) if b]
    assert len(bodies) == 1, f'{kernel}: {len(bodies)} definitions'
    assert ways_out_without_wait(bodies[0]) == []


def test_the_check_sees_a_missing_wait():
    ok = '{ if (!early) grid_dep_wait(); if (x) { grid_dep_wait(); return; } if (warp == 8) { load(); grid_dep_wait(); } if (y) return; }'
    assert ways_out_without_wait(ok) == []
    assert ways_out_without_wait(ok.replace('x) { grid_dep_wait();', 'x) {')) == ['return in if (x)']
    assert ways_out_without_wait(ok.replace('warp == 8', 'z')) == ['if (y) return in the kernel', 'end of the kernel']
    assert ways_out_without_wait('{ auto f = [&](int i) { if (i) return; g(); }; grid_dep_wait(); }') == []


def _stops():
    return [(f, m.group(1)) for f, t in SOURCES.items() for m in re.finditer(r'\bs_abort = ([^;]+);', t)]


@pytest.mark.parametrize('name,value', _stops())
def test_a_set_error_word_stops_the_ctas_that_start_later(name, value):
    """A CTA reads the error word before its first wait, so that one wait that has run out does not cost every CTA its limit.  A CTA that
    may run beside the kernel that clears the word cannot read it: that is a matter of its place in the grid, never of the launch."""
    m = re.fullmatch(r'(?:(\w+) \? 0 : )?\*\(volatile int\*\)err', value)
    assert m, f'{name}: s_abort = {value}'
    if m.group(1):
        rule = re.search(r'const bool ' + m.group(1) + r' = ([^;]+);', SOURCES[name]).group(1)
        assert 'blockIdx' in rule, f'{name}: {m.group(1)} = {rule}'
        assert f'if (!{m.group(1)}) grid_dep_wait();' in SOURCES[name]


def test_the_stop_is_looked_for_where_it_is():
    assert {f for f, _ in _stops()} >= {'nha_chunk_state_umma.cu', 'nha_chunk_fwd_pipe.cu'}
